// tcgen05 / TMEM / TMA reverse pass of triangle attention for sm_100a (f16 and bf16, head_dim 32).
//
// Replaces the reference's Triton kernels `_backward_preprocess`, `_backward_query`,
// `_backward_key_value` and `_backward_shared_bias` (oops/attention/triangle/triton/kernel.py:374-873).
// With P = exp(S - lse), dP = dO V^T, dS = P o (dP - delta) (kernel.py:499-564):
//
//   delta kernel     delta[q] = sum_d O[q,d] dO[q,d]                           (memory bound)
//   dQ kernel        CTA = (batch,row,head, one 128-query tile), streams 64-key steps:
//                    S = Q K^T, dP = dO V^T -> dS (16-bit, back into tensor memory) -> dQ += dS K.
//                    A per-row bias gradient is dS itself and is stored from here.
//   dK/dV kernel     CTA = (batch,row,head, one 128-key tile), streams 64-query steps, transposed:
//                    S^T = K Q^T, dP^T = V dO^T -> P^T, dS^T (tensor memory) -> dV += P^T dO, dK += dS^T Q.
//                    It reads a transposed copy of the bias so that a thread (= one key) reads a bias row.
//   shared-bias      CTA = (row part, batch, head, query tile, key tile) loops over its rows:
//   gradient         S, dP -> dS accumulated in f32 registers over the rows (four warpgroups split the
//                    128 keys), one f32 partial plane per part; a last kernel adds the parts in a fixed
//                    order (no atomics, bitwise reproducible).
//
// All kernels share the forward kernel's structure: one TMA producer thread, one MMA-issuing thread,
// warpgroups of 128 threads that own one tensor-memory lane (= one query or key) each.  The dQ and dK/dV
// kernels keep 256 tensor-memory columns and under 113 KB of shared memory, so two CTAs share an SM: their
// MMA threads run independently and one CTA's prologue and epilogue overlap the other's steps.
#include <type_traits>

#include "ta_tensor_common.cuh"

namespace oops_ta {
namespace {

using namespace ptx;

constexpr int kTilesPerCta = 1;                          // dQ and dK/dV kernels: 128-row tiles owned by one CTA (1 or 2)
constexpr int kElemWarps = 8 * kTilesPerCta;             // two warpgroups per tile
constexpr int kThreads = (kElemWarps + (kTilesPerCta == 2 ? 3 : 2)) * 32;
constexpr int kCtasPerSm = kTilesPerCta == 2 ? 1 : 2;
constexpr int kDbElemWarps = 16;                         // shared-bias kernel: one warpgroup per 32 of the tile's 128 keys
constexpr int kDbThreads = (kDbElemWarps + 2) * 32;
constexpr int kStep = 64;                               // streamed keys (dQ) or queries (dK/dV) per step
constexpr int kBigTile = kTile * kHeadDim * 2;          // 8 KiB: 128 x 32 tile
constexpr int kSmallTile = kStep * kHeadDim * 2;        // 4 KiB: 64 x 32 tile
constexpr int kBiasStep = kTile * kStep * 2;            // 16 KiB: 128 x 64 bias tile (one swizzle-128 box)
constexpr int kRing = 4;                                // ring depth of the streamed operand pairs

// ---------------------------------------------------------------------------------------------
// small helper kernels
// ---------------------------------------------------------------------------------------------

// delta[b][r][h][q] = sum_d O * dO.  Four lanes share a cell and take its heads four at a time: a warp's loads cover eight cells, 64 bytes of
// a head each, and the lanes end with a head's sum each.  `row_inner`: cells of
// neighbouring rows, not columns, are neighbours in memory (the ending-node form).  The first blocks look at
// the mask: live[b][r] has bit k set when some key of columns 128 k .. 128 k + 127 of the row is kept, the
// second word of a row whether all of them are, the third how many keys a row keeps if these are its first ones (else ~0), and
// behind the rows' words one word per eight rows tells whether they drop any key.
// Bound by HBM.  With a (cell, head) per four lanes the divisions that place it were as many instructions as HBM had time for, and the
// mask's blocks, last in the grid and a load at a time, ran on alone.  N = 256, two samples: 18.4 -> 11.7 us; N = 768: 71.8 -> 50.3 us
// (302 MB of tensors and 9 of sums: 6.2 TB/s of the copy's 6.56).
// HEADS == 1: one head, whose group would be three idle loads and whose registers would halve the CTAs of an SM (N = 256: 3.8 us, as a group 5.3).
template <typename T, int HEADS>
__global__ void __launch_bounds__(256, HEADS == 1 ? 6 : 4) prepare_kernel(oops_ta_pair out, oops_ta_pair dout, float* delta, uint32_t cells, int cols,
                                                      int heads, int rows, int vec_ok, int row_inner, uint32_t mask_blocks,
                                                      const uint8_t* mask, int64_t m_sb, int64_t m_sr, int64_t m_sc,
                                                      uint32_t* live, int num_rows) {
  if (blockIdx.x < mask_blocks) {
    const int block = int(blockIdx.x), row = block * 8 + int(threadIdx.x >> 5), lane = threadIdx.x & 31;
    bool dropped = false;
    if (row < num_rows) {
      const uint8_t* bytes = mask + (row / rows) * m_sb + int64_t(row % rows) * m_sr;
      uint32_t bits = 0, full = 0;
      int count = 0, end = 0;  // kept keys, and one behind the last of them
      constexpr int kBatch = 16;  // words of 32 keys whose bytes travel together
      for (int first = 0; first < cols; first += kBatch * 32) {
        uint32_t kept[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int key = first + i * 32 + lane;
          kept[i] = key < cols ? ldg_u8_here(bytes + int64_t(key) * m_sc) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) kept[i] = __ballot_sync(0xffffffffu, kept[i] != 0);
#pragma unroll
        for (int tile = 0; tile < kBatch / 4; ++tile) {
          uint32_t any = 0;
          int wanted = 0, found = 0;
#pragma unroll
          for (int i = 4 * tile; i < 4 * tile + 4; ++i) {
            any |= kept[i];
            found += __popc(kept[i]);
            wanted += min(32, max(0, cols - (first + i * 32)));
            if (kept[i] != 0) end = first + i * 32 + 32 - __clz(int(kept[i]));
          }
          count += found;
          if (wanted == 0) break;
          if (any != 0) bits |= 1u << (first / 128 + tile);
          if (found == wanted) full |= 1u << (first / 128 + tile);
          else dropped = true;
        }
      }
      if (lane == 0) {
        live[row] = bits;
        live[num_rows + row] = full;
        live[2 * num_rows + row] = count == end ? uint32_t(count) : ~0u;
      }
    }
    const int drops = __syncthreads_or(dropped);
    if (threadIdx.x == 0) live[3 * num_rows + block] = uint32_t(drops != 0);
    return;
  }
  const uint32_t cell = (blockIdx.x - mask_blocks) * 64u + (threadIdx.x >> 2);
  const int part = threadIdx.x & 3;
  const bool there = cell < cells;  // (a warp's lanes stay together for the exchange)
  const uint32_t inner = row_inner ? uint32_t(rows) : uint32_t(cols), outer = row_inner ? uint32_t(cols) : uint32_t(rows);
  const uint32_t i = cell % inner, rest = cell / inner, o = rest % outer, b = rest / outer;
  const uint32_t r = row_inner ? i : o, q = row_inner ? o : i;
  const T* po = reinterpret_cast<const T*>(out.ptr) + b * out.sb + int64_t(r) * out.sr + int64_t(q) * out.sc + part * 8;
  const T* pd = reinterpret_cast<const T*>(dout.ptr) + b * dout.sb + int64_t(r) * dout.sr + int64_t(q) * dout.sc + part * 8;
  float* to = delta + (int64_t(b) * rows + r) * heads * cols + q;
  for (int h0 = 0; h0 < heads; h0 += HEADS) {
    float dot[HEADS] = {};
    if (vec_ok) {
      uint4 a[HEADS], g[HEADS];
#pragma unroll
      for (int n = 0; n < HEADS; ++n) {
        const bool take = there && h0 + n < heads;
        a[n] = ldg_v4_here_if(po + int64_t(h0 + n) * out.sh, take);
        g[n] = ldg_v4_here_if(pd + int64_t(h0 + n) * dout.sh, take);
      }
#pragma unroll
      for (int n = 0; n < HEADS; ++n) {
        const uint32_t aw[4] = {a[n].x, a[n].y, a[n].z, a[n].w}, gw[4] = {g[n].x, g[n].y, g[n].z, g[n].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) dot[n] += Half2<T>::lo(aw[e]) * Half2<T>::lo(gw[e]) + Half2<T>::hi(aw[e]) * Half2<T>::hi(gw[e]);
      }
    } else if (there) {
#pragma unroll
      for (int n = 0; n < HEADS; ++n) {
        if (h0 + n >= heads) break;
#pragma unroll
        for (int c = 0; c < 8; ++c) dot[n] += float(po[int64_t(h0 + n) * out.sh + c]) * float(pd[int64_t(h0 + n) * dout.sh + c]);
      }
    }
    float own = 0.f;
#pragma unroll
    for (int n = 0; n < HEADS; ++n) {
      dot[n] += __shfl_xor_sync(0xffffffffu, dot[n], 1);
      dot[n] += __shfl_xor_sync(0xffffffffu, dot[n], 2);
      if (n == part) own = dot[n];
    }
    if (there && part < HEADS && h0 + part < heads) to[int64_t(h0 + part) * cols] = own;
  }
}

// Whether the mask that prepare_kernel has looked at keeps every key (one warp's answer).
__device__ __forceinline__ bool keeps_all(const uint32_t* live, int num_rows, int lane) {
  const int words = (num_rows + 7) / 8;
  bool drops = false;
#pragma unroll 4
  for (int i = lane; i < words; i += 32) drops |= __ldg(live + 3 * num_rows + i) != 0;
  return !__any_sync(0xffffffffu, drops);
}

// dst[z][k][q] = src[z][q][k] for 16-bit elements; dst rows are `dst_stride` elements apart.
__global__ void transpose_bias_kernel(const uint16_t* src, uint16_t* dst, int cols, int64_t s_q, int64_t s_h, int64_t s_g,
                                      int64_t s_b, int heads, int groups, int64_t dst_stride) {
  __shared__ uint16_t tile[32][34];
  const int z = blockIdx.z;
  const int h = z % heads;
  const int g = (z / heads) % groups;
  const int64_t b = z / (heads * groups);
  const uint16_t* plane = src + b * s_b + g * s_g + h * s_h;
  uint16_t* out = dst + int64_t(z) * cols * dst_stride;
  const int k0 = blockIdx.x * 32, q0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int q = q0 + i, k = k0 + threadIdx.x;
    tile[i][threadIdx.x] = (q < cols && k < cols) ? plane[int64_t(q) * s_q + k] : uint16_t(0);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int k = k0 + i, q = q0 + threadIdx.x;
    if (k < cols && q < dst_stride) out[int64_t(k) * dst_stride + q] = q < cols ? tile[threadIdx.x][i] : uint16_t(0);
  }
}

// dbias = the sum of its parts in their order.  `quads`: a thread takes four keys, whose rows are whole 16-byte words (N = 256, two
// samples: 9.2 -> 5.0 us; the ragged sample of 700 tokens: 45.8 -> 11.9).
template <typename T>
__global__ void __launch_bounds__(256) reduce_parts_kernel(const float* parts, int num_parts, void* dbias, int64_t sb, int64_t sh, int64_t sq,
                                                           int64_t sk, int heads, int cols, int64_t plane, int quads) {
  const int64_t at = int64_t(blockIdx.x) * 256 + threadIdx.x, i = quads ? at * 4 : at;
  if (i >= plane) return;
  const int64_t row = i / cols;  // (batch, head, query)
  const int k = int(i - row * cols), q = int(row % cols), h = int(row / cols % heads);
  T* to = reinterpret_cast<T*>(dbias) + row / cols / heads * sb + h * sh + int64_t(q) * sq + int64_t(k) * sk;
  if (quads) {
    float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int p = 0; p < num_parts; ++p) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(parts + int64_t(p) * plane + i));
      total = make_float4(total.x + v.x, total.y + v.y, total.z + v.z, total.w + v.w);
    }
    if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(to) = total;
    else *reinterpret_cast<uint2*>(to) = make_uint2(Half2<T>::pack(total.x, total.y), Half2<T>::pack(total.z, total.w));
  } else {
    float total = 0.f;
#pragma unroll 4
    for (int p = 0; p < num_parts; ++p) total += __ldg(parts + int64_t(p) * plane + i);
    *to = T(total);
  }
}

// 16-bit row store of 32 channels from f32 accumulator words, scaled.
template <typename T>
__device__ __forceinline__ void store_row32(T* dst, const uint32_t (&acc)[32], float scale, bool vec_ok) {
  uint32_t o2[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    o2[i] = Half2<T>::pack(__uint_as_float(acc[2 * i]) * scale, __uint_as_float(acc[2 * i + 1]) * scale);
  if (vec_ok) {
    uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int i = 0; i < 4; ++i) d4[i] = make_uint4(o2[4 * i], o2[4 * i + 1], o2[4 * i + 2], o2[4 * i + 3]);
  } else {
    unsigned short* d0 = reinterpret_cast<unsigned short*>(dst);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      d0[2 * i] = (unsigned short)(o2[i] & 0xffffu);
      d0[2 * i + 1] = (unsigned short)(o2[i] >> 16);
    }
  }
}

__device__ __forceinline__ bool pair_vec_ok(const oops_ta_pair& t) {
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 8 == 0 && t.sr % 8 == 0 && t.sc % 8 == 0 && t.sh % 8 == 0;
}

// ---------------------------------------------------------------------------------------------
// shared pieces of the three tensor kernels
// ---------------------------------------------------------------------------------------------
// The single-pass kernel has 640 threads: warps 0-15 are four warpgroups of 128 threads that do the element-wise work, warp 16 is
// the TMA producer, warp 17 issues the score products (S, dP) and owns the tensor-memory allocation, warp 18
// issues the accumulating products (dQ, or dK and dV), warp 19 prepares statistics and masked tiles; the shared-bias kernel has neither.  Two issuing
// threads keep the tensor core fed: neither kind of product waits behind the other's barrier.  The element-wise
// work of the reverse pass has no reduction along a score row, so the 64 columns of a step are split
// between two warpgroups that address the same tensor-memory lanes (warp % 4 selects the lanes).

constexpr int kProducerWarp = kElemWarps, kMmaWarp = kElemWarps + 1, kAccWarp = kElemWarps + 2;
constexpr int kDbProducerWarp = kDbElemWarps, kDbMmaWarp = kDbElemWarps + 1;

constexpr int kMaxKeepWords = 512;  // keep-bit table: one bit per key column, cols <= 16384

// Eight columns of the reverse-pass element math on packed f32 pairs:
//   p  = 2^(s * (scale*log2e) + bias * log2e + nl)        nl = -lse * log2e
//   ds = p * (dp + nd)                                     nd = -delta
// sraw/draw are the tensor-memory words of S and dP (adjacent columns form a pair), bias_chunk points at
// eight 16-bit bias values, nl2/nd2 hold the four (nl, nl') and (nd, nd') pairs of these columns.
template <typename T, bool HAS_BIAS>
__device__ __forceinline__ void score_grad8(const uint32_t* sraw, const uint32_t* draw, const uint8_t* bias_chunk, f32x2 c2,
                                            f32x2 log2e2, const f32x2* nl2, const f32x2* nd2, f32x2* p2, f32x2* ds2) {
  uint32_t bw[4] = {0, 0, 0, 0};
  if (HAS_BIAS) {
    const uint4 v = *reinterpret_cast<const uint4*>(bias_chunk);
    bw[0] = v.x; bw[1] = v.y; bw[2] = v.z; bw[3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const f32x2 s2 = pack2(__uint_as_float(sraw[2 * i]), __uint_as_float(sraw[2 * i + 1]));
    const f32x2 d2 = pack2(__uint_as_float(draw[2 * i]), __uint_as_float(draw[2 * i + 1]));
    const f32x2 offset = HAS_BIAS ? fma2(Half2<T>::widen(bw[i]), log2e2, nl2[i]) : nl2[i];
    float lo, hi;
    unpack2(fma2(s2, c2, offset), lo, hi);
    const f32x2 p = pack2(ex2(lo), ex2(hi));
    p2[i] = p;
    ds2[i] = mul2(p, add2(d2, nd2[i]));
  }
}

// Same with the eight bias values already in registers (four packed words).
template <typename T, bool HAS_BIAS>
__device__ __forceinline__ void score_grad8_words(const uint32_t* sraw, const uint32_t* draw, const uint4 bias_words, f32x2 c2,
                                                  f32x2 log2e2, f32x2 nl, f32x2 nd, f32x2* p2, f32x2* ds2) {
  const uint32_t bw[4] = {bias_words.x, bias_words.y, bias_words.z, bias_words.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const f32x2 s2 = pack2(__uint_as_float(sraw[2 * i]), __uint_as_float(sraw[2 * i + 1]));
    const f32x2 d2 = pack2(__uint_as_float(draw[2 * i]), __uint_as_float(draw[2 * i + 1]));
    const f32x2 offset = HAS_BIAS ? fma2(Half2<T>::widen(bw[i]), log2e2, nl) : nl;
    float lo, hi;
    unpack2(fma2(s2, c2, offset), lo, hi);
    const f32x2 p = pack2(ex2(lo), ex2(hi));
    p2[i] = p;
    ds2[i] = mul2(p, add2(d2, nd));
  }
}

__device__ __forceinline__ f32x2 select2(f32x2 v, uint32_t bits, int at) {
  float lo, hi;
  unpack2(v, lo, hi);
  if (((bits >> at) & 1u) == 0) lo = 0.f;
  if (((bits >> (at + 1)) & 1u) == 0) hi = 0.f;
  return pack2(lo, hi);
}

template <typename T>
__device__ __forceinline__ uint32_t pack16(f32x2 v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return Half2<T>::pack(lo, hi);
}

// ---------------------------------------------------------------------------------------------
// dQ kernel
// ---------------------------------------------------------------------------------------------

struct DqSmem {
  static constexpr int q = 0;                                         // [tiles] 128 x 32
  static constexpr int dout = q + kTilesPerCta * kBigTile;            // [tiles] 128 x 32
  static constexpr int kv = dout + kTilesPerCta * kBigTile;           // [kRing] K step (4 KiB) + V step (4 KiB)
  static constexpr int bias = kv + kRing * 2 * kSmallTile;            // [tiles][2 buffers] 128 x 64
  static constexpr int bars = bias + 2 * kTilesPerCta * kBiasStep;
  static constexpr int qd_full = 0;                      // [2]
  static constexpr int kv_full = qd_full + 2;            // [kRing]
  static constexpr int kv_empty = kv_full + kRing;       // [kRing]
  static constexpr int k_ready = kv_empty + kRing;       // [kRing]
  static constexpr int bias_full = k_ready + kRing;      // [4]
  static constexpr int bias_empty = bias_full + 4;       // [4]
  static constexpr int sd_full = bias_empty + 4;         // [2] S and dP of a step are in tensor memory
  static constexpr int sd_free = sd_full + 2;            // [2] both have been read into registers
  static constexpr int ds_full = sd_free + 2;            // [2] dS (16-bit) is in tensor memory
  static constexpr int ds_done = ds_full + 2;            // [2] the dQ product has consumed it
  static constexpr int dq_done = ds_done + 2;            // [2] last dQ product finished
  static constexpr int num_bars = dq_done + 2;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int drop_flags = abort_flag + 4;  // [<= 16] per-warp: the mask drops a key of this row
  static constexpr int keep = drop_flags + 64;
  static constexpr int total = keep + kMaxKeepWords * 4;
};
constexpr int kDqSmemBytes = DqSmem::total + 1024;

struct DqParams {
  CUtensorMap map_q, map_dout, map_k, map_v, map_bias;
  oops_ta_pair dq;
  const float* lse;
  const float* delta;
  const uint8_t* mask;
  int64_t m_sb, m_sr, m_sc;
  void* dbias_rows;  // per-row bias gradient (may be null)
  int64_t db_sb, db_sg, db_sh, db_sq, db_sk;
  int batch, rows, cols, heads, bias_groups;
  int q_pairs, k_steps;
  int write_dq;
  float scale;
};

template <typename T, bool HAS_BIAS>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) ta_bwd_dq_kernel(const __grid_constant__ DqParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + DqSmem::abort_flag);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + DqSmem::tmem_slot);
  uint32_t* keep_words = reinterpret_cast<uint32_t*>(smem_gen + DqSmem::keep);
  auto bar = [&](int index) -> uint32_t { return smem_base + DqSmem::bars + index * 8; };

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (device_failed()) return;
  int idx = blockIdx.x;
  const int qp = idx % P.q_pairs;
  idx /= P.q_pairs;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int r = idx % P.rows;
  const int b = idx / P.rows;
  const int q0 = qp * kTilesPerCta * kTile;
  const int n_tiles = (kTilesPerCta == 2 && q0 + kTile < P.cols) ? 2 : 1;
  const int KS = P.k_steps;
  const int g = P.bias_groups == 1 ? 0 : r;
  const bool has_mask = P.mask != nullptr;
  const bool has_bits = has_mask || (P.cols % kStep) != 0;
  // tensor-memory columns of query tile w: S [0,64) | dP [64,128) | dS [128,160) | dQ [160,192)
  constexpr int kTileCols = 192, kDpCol = 64, kDsCol = 128, kDqCol = 160;
  constexpr int kTmemCols = kTilesPerCta == 2 ? 512 : 256;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kTilesPerCta; ++i) {
      mbar_init(bar(DqSmem::qd_full + i), 1);
      mbar_init(bar(DqSmem::sd_full + i), 1);
      mbar_init(bar(DqSmem::sd_free + i), 8);
      mbar_init(bar(DqSmem::ds_full + i), 8);
      mbar_init(bar(DqSmem::ds_done + i), 1);
      mbar_init(bar(DqSmem::dq_done + i), 1);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(bar(DqSmem::kv_full + i), 1);
      mbar_init(bar(DqSmem::kv_empty + i), 1);
      mbar_init(bar(DqSmem::k_ready + i), 4);
    }
    for (int i = 0; i < 2 * kTilesPerCta; ++i) {
      mbar_init(bar(DqSmem::bias_full + i), 1);
      mbar_init(bar(DqSmem::bias_empty + i), 8);
    }
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_base + DqSmem::tmem_slot, kTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // The keep-bit table is built after the CTA-wide barrier, by the element-wise warps, while the producer's first
  // copies are already in flight; only its users (those warps and the issuing warps) meet at a named barrier.
  uint32_t* drop_flags = reinterpret_cast<uint32_t*>(smem_gen + DqSmem::drop_flags);
  bool signoff = false;
  if (has_bits && warp != kProducerWarp) {
    if (warp < kElemWarps) {
      const uint8_t* mask_row = has_mask ? P.mask + b * P.m_sb + int64_t(r) * P.m_sr : nullptr;
      bool dropped_any = false;
      for (int word = warp; word < KS * 2; word += kElemWarps) {
        const int key = word * 32 + lane;
        bool keep = key < P.cols;
        if (keep && has_mask) {
          keep = mask_row[int64_t(key) * P.m_sc] != 0;
          dropped_any |= !keep;
        }
        const uint32_t bits = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) keep_words[word] = bits;
      }
      dropped_any = __any_sync(0xffffffffu, dropped_any);
      if (lane == 0) drop_flags[warp] = dropped_any ? 1u : 0u;
    }
    named_barrier_sync(1, kThreads - 32);
    // Key rows only need the sign-off handshake when the mask really drops a key of this row.
    if (has_mask) {
#pragma unroll
      for (int i = 0; i < kElemWarps; ++i) signoff |= drop_flags[i] != 0;
    }
  }

  if (warp == kProducerWarp) {
    if (lane == 0) {
      bool ok = true;
      for (int w = 0; w < n_tiles; ++w) {
        mbar_expect_tx(bar(DqSmem::qd_full + w), 2 * kBigTile);
        tma_load_5d(smem_base + DqSmem::q + w * kBigTile, &P.map_q, bar(DqSmem::qd_full + w), 0, h, q0 + w * kTile, r, b);
        tma_load_5d(smem_base + DqSmem::dout + w * kBigTile, &P.map_dout, bar(DqSmem::qd_full + w), 0, h, q0 + w * kTile, r, b);
      }
      for (int j = 0; j < KS && ok; ++j) {
        const int st = j % kRing, round = j / kRing;
        if (j >= kRing) ok = mbar_wait(bar(DqSmem::kv_empty + st), (round - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(DqSmem::kv_full + st), 2 * kSmallTile);
        const uint32_t dst = smem_base + DqSmem::kv + st * 2 * kSmallTile;
        tma_load_5d(dst, &P.map_k, bar(DqSmem::kv_full + st), 0, h, j * kStep, r, b);
        tma_load_5d(dst + kSmallTile, &P.map_v, bar(DqSmem::kv_full + st), 0, h, j * kStep, r, b);
        if (HAS_BIAS) {
          for (int w = 0; w < n_tiles && ok; ++w) {
            const int slot = w * 2 + (j & 1);
            if (j >= 2) ok = mbar_wait(bar(DqSmem::bias_empty + slot), ((j >> 1) - 1) & 1, abort_flag);
            if (!ok) break;
            mbar_expect_tx(bar(DqSmem::bias_full + slot), kBiasStep);
            tma_load_5d(smem_base + DqSmem::bias + slot * kBiasStep, &P.map_bias, bar(DqSmem::bias_full + slot), j * kStep,
                        q0 + w * kTile, h, g, b);
          }
        }
      }
    }
  } else if (warp == kMmaWarp || (kTilesPerCta == 2 && warp == kAccWarp)) {
    // One tile per CTA: one thread issues everything in the order the events arrive (scores of step j+1 when the
    // warpgroups have read step j, dQ of step j when they have stored dS).  Two tiles per CTA: a second thread issues
    // the dQ products, so that neither kind of product waits behind the other tile's barrier.
    if (lane == 0) {
      constexpr uint32_t fmt = Half2<T>::kFormat;
      constexpr uint32_t idesc_s = instr_desc(fmt, 0, 0, kTile, kStep);
      constexpr uint32_t idesc_dq = instr_desc(fmt, 0, 1, kTile, kHeadDim);
      const bool do_scores = warp == kMmaWarp, do_acc = kTilesPerCta == 1 || warp == kAccWarp;
      bool ok = true;
      // a K/V step is usable once the copy has landed and, with a mask, once warpgroup 0 has signed it off
      auto wait_step = [&](int j) -> bool {
        bool ready = mbar_wait(bar(DqSmem::kv_full + j % kRing), (j / kRing) & 1, abort_flag);
        if (ready && signoff) ready = mbar_wait(bar(DqSmem::k_ready + j % kRing), (j / kRing) & 1, abort_flag);
        return ready;
      };
      // S = Q K^T and dP = dO V^T of step j for query tile w (all operands K-major, 64-byte swizzle)
      auto issue_scores = [&](int j, int w) {
        // the bias tile of the step has landed before the scores are announced: the warpgroups do not wait for it
        if (HAS_BIAS && !mbar_wait(bar(DqSmem::bias_full + w * 2 + (j & 1)), (j >> 1) & 1, abort_flag)) return;
        const uint32_t kv = smem_base + DqSmem::kv + (j % kRing) * 2 * kSmallTile;
        const uint32_t s_t = tmem_base + w * kTileCols;
        const uint64_t qdesc = smem_desc(smem_base + DqSmem::q + w * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t ddesc = smem_desc(smem_base + DqSmem::dout + w * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t kdesc = smem_desc(kv, 16, 512, kSwizzle64B);
        const uint64_t vdesc = smem_desc(kv + kSmallTile, 16, 512, kSwizzle64B);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(s_t, qdesc + uint64_t(kk * 2), kdesc + uint64_t(kk * 2), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(s_t + kDpCol, ddesc + uint64_t(kk * 2), vdesc + uint64_t(kk * 2), idesc_s, kk > 0 ? 1u : 0u);
        mma_commit(bar(DqSmem::sd_full + w));
      };
      // dQ[128 x 32] += dS[128 x 64] K[64 x 32]; K is MN-major (channel contiguous).
      auto issue_dq = [&](int j, int w) {
        const int st = j % kRing;
        const uint32_t tile_t = tmem_base + w * kTileCols;
        const uint64_t kdesc = smem_desc(smem_base + DqSmem::kv + st * 2 * kSmallTile, 16, 512, kSwizzle64B);
#pragma unroll
        for (int kk = 0; kk < kStep / 16; ++kk)
          mma_ts(tile_t + kDqCol, tile_t + kDsCol + kk * 8, kdesc + uint64_t(kk * (1024 >> 4)), idesc_dq,
                 (j > 0 || kk > 0) ? 1u : 0u);
        mma_commit(bar(DqSmem::ds_done + w));
        if (j == KS - 1) mma_commit(bar(DqSmem::dq_done + w));
        if (w == n_tiles - 1) mma_commit(bar(DqSmem::kv_empty + st));
      };
      if (do_scores) {
        for (int w = 0; w < n_tiles && ok; ++w) ok = mbar_wait(bar(DqSmem::qd_full + w), 0, abort_flag);
        if (ok) ok = wait_step(0);
        if (ok) {
          tc_fence_after_sync();
          for (int w = 0; w < n_tiles; ++w) issue_scores(0, w);
        }
      }
      for (int j = 0; j < KS && ok; ++j) {
        if (do_scores && j + 1 < KS) {
          ok = wait_step(j + 1);
          for (int w = 0; w < n_tiles && ok; ++w) {
            ok = mbar_wait(bar(DqSmem::sd_free + w), j & 1, abort_flag);
            if (!ok) break;
            tc_fence_after_sync();
            issue_scores(j + 1, w);
          }
        }
        if (do_acc && ok) {
          if (!do_scores) ok = wait_step(j);
          for (int w = 0; w < n_tiles && ok; ++w) {
            ok = mbar_wait(bar(DqSmem::ds_full + w), j & 1, abort_flag);
            if (!ok) break;
            tc_fence_after_sync();
            issue_dq(j, w);
          }
        }
      }
    }
  } else if (warp < kElemWarps && (warp >> 3) < n_tiles) {
    const int w = warp >> 3;          // query tile
    const int half = (warp >> 2) & 1; // which 32 of the step's 64 keys
    const int t = tid & (kTile - 1);
    const uint32_t lane_field = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tile_t = tmem_base + lane_field + w * kTileCols;
    const int q_index = q0 + w * kTile + t;
    const bool q_valid = q_index < P.cols;
    const int64_t stat_at = ((int64_t(b) * P.rows + r) * P.heads + h) * P.cols + q_index;
    const float neg_lse2 = q_valid ? -P.lse[stat_at] * kLog2e : -INFINITY;
    const float delta = q_valid ? P.delta[stat_at] : 0.f;
    const float scale = P.scale;
    const f32x2 c2 = pack2(scale * kLog2e, scale * kLog2e), log2e2 = pack2(kLog2e, kLog2e);
    const f32x2 nl2[4] = {pack2(neg_lse2, neg_lse2), pack2(neg_lse2, neg_lse2), pack2(neg_lse2, neg_lse2), pack2(neg_lse2, neg_lse2)};
    const f32x2 nd2[4] = {pack2(-delta, -delta), pack2(-delta, -delta), pack2(-delta, -delta), pack2(-delta, -delta)};
    T* db_row = nullptr;
    bool db_vec = false;
    if (P.dbias_rows && q_valid) {
      db_row = reinterpret_cast<T*>(P.dbias_rows) + b * P.db_sb + int64_t(r) * P.db_sg + h * P.db_sh + int64_t(q_index) * P.db_sq;
      db_vec = P.db_sk == 1 && (reinterpret_cast<uintptr_t>(db_row) & 15) == 0;
    }
    bool ok = true;

    for (int j = 0; j < KS && ok; ++j) {
      uint32_t my_bits = 0xffffffffu;
      bool step_all_kept = true;
      if (has_bits) {
        const uint2 wds = *reinterpret_cast<const uint2*>(keep_words + j * 2);
        my_bits = half ? wds.y : wds.x;
        step_all_kept = (wds.x & wds.y) == 0xffffffffu;
        if (signoff && warp < 4) {
          // Key rows of dropped keys must not reach the dQ product (0 * inf): clear them in shared memory.
          const int st = j % kRing;
          if (!step_all_kept) {
            ok = mbar_wait(bar(DqSmem::kv_full + st), (j / kRing) & 1, abort_flag);
            if (!ok) break;
            const uint32_t word = (t < 32) ? wds.x : wds.y;
            if (t < kStep && ((word >> (t & 31)) & 1u) == 0) {
              uint4* row = reinterpret_cast<uint4*>(smem_gen + DqSmem::kv + st * 2 * kSmallTile + t * 64);
              row[0] = row[1] = row[2] = row[3] = make_uint4(0, 0, 0, 0);
            }
            fence_proxy_async_smem();
          }
          mbar_arrive_warp(bar(DqSmem::k_ready + st));
        }
      }
      ok = mbar_wait(bar(DqSmem::sd_full + w), j & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sraw[32], draw[32];
      tmem_ld32(tile_t + half * 32, sraw);
      tmem_ld32(tile_t + kDpCol + half * 32, draw);
      tmem_wait_ld();
      tmem_loaded(sraw);
      tmem_loaded(draw);
      tc_fence_before_sync();
      mbar_arrive_warp(bar(DqSmem::sd_free + w));
      const int slot = w * 2 + (j & 1);
      const uint8_t* bias_row = smem_gen + DqSmem::bias + slot * kBiasStep + t * 128 + (((t & 7) ^ (half * 4)) << 4);
      uint32_t packed[16];
      const int key0 = j * kStep + half * 32;
#pragma unroll
      for (int i8 = 0; i8 < 4; ++i8) {
        f32x2 p2[4], ds2[4];
        score_grad8<T, HAS_BIAS>(sraw + i8 * 8, draw + i8 * 8, swizzled_chunk(bias_row, i8), c2, log2e2, nl2,
                                 nd2, p2, ds2);
        if (my_bits != 0xffffffffu) {
#pragma unroll
          for (int i = 0; i < 4; ++i) ds2[i] = select2(ds2[i], my_bits, i8 * 8 + 2 * i);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) packed[i8 * 4 + i] = pack16<T>(ds2[i]);
        if (db_row) {
          if (db_vec && key0 + 32 <= P.cols) {
            *reinterpret_cast<uint4*>(db_row + key0 + i8 * 8) =
                make_uint4(packed[i8 * 4], packed[i8 * 4 + 1], packed[i8 * 4 + 2], packed[i8 * 4 + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float lo, hi;
              unpack2(ds2[i], lo, hi);
              if (key0 + i8 * 8 + 2 * i < P.cols) db_row[int64_t(key0 + i8 * 8 + 2 * i) * P.db_sk] = T(lo);
              if (key0 + i8 * 8 + 2 * i + 1 < P.cols) db_row[int64_t(key0 + i8 * 8 + 2 * i + 1) * P.db_sk] = T(hi);
            }
          }
        }
      }
      if (HAS_BIAS) mbar_arrive_warp(bar(DqSmem::bias_empty + slot));
      if (j > 0) {
        // the dQ product of the previous step must have finished reading the dS columns
        ok = mbar_wait(bar(DqSmem::ds_done + w), (j - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
      }
      tmem_st16(tile_t + kDsCol + half * 16, packed);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive_warp(bar(DqSmem::ds_full + w));
    }

    if (ok) ok = mbar_wait(bar(DqSmem::dq_done + w), 0, abort_flag);
    if (ok && half == 0) {
      tc_fence_after_sync();
      uint32_t acc[32];
      tmem_ld32(tile_t + kDqCol, acc);
      tmem_wait_ld();
      tmem_loaded(acc);
      if (q_valid && P.write_dq) {
        T* dst = reinterpret_cast<T*>(P.dq.ptr) + b * P.dq.sb + int64_t(r) * P.dq.sr + int64_t(q_index) * P.dq.sc + h * P.dq.sh;
        store_row32<T>(dst, acc, scale, pair_vec_ok(P.dq));
      }
    }
  }
  teardown(abort_flag, tmem_base, kMmaWarp, kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// dK / dV kernel (transposed: a thread owns a key)
// ---------------------------------------------------------------------------------------------

struct DkvSmem {
  static constexpr int k = 0;                                          // [tiles] 128 x 32
  static constexpr int v = k + kTilesPerCta * kBigTile;                // [tiles] 128 x 32
  static constexpr int qd = v + kTilesPerCta * kBigTile;               // [kRing] Q step (4 KiB) + dO step (4 KiB)
  static constexpr int bias = qd + kRing * 2 * kSmallTile;             // [tiles][2 buffers] 128 keys x 64 queries
  static constexpr int stats = bias + 2 * kTilesPerCta * kBiasStep;    // [warps][2 buffers][64 floats]: -lse*log2e | -delta
  static constexpr int bars = stats + 2 * kElemWarps * 256;
  static constexpr int kv_full = 0;                      // [2]
  static constexpr int qd_full = kv_full + 2;            // [kRing]
  static constexpr int qd_empty = qd_full + kRing;       // [kRing]
  static constexpr int bias_full = qd_empty + kRing;     // [4]
  static constexpr int bias_empty = bias_full + 4;       // [4]
  static constexpr int sd_full = bias_empty + 4;         // [2] S^T and dP^T of a step are in tensor memory
  static constexpr int sd_free = sd_full + 2;            // [2] both have been read into registers
  static constexpr int pds_full = sd_free + 2;           // [2] P^T and dS^T (16-bit) are in tensor memory
  static constexpr int pds_done = pds_full + 2;          // [2] the dV / dK products have consumed them
  static constexpr int done = pds_done + 2;              // [2]
  static constexpr int num_bars = done + 2;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int total = abort_flag + 4;
};
constexpr int kDkvSmemBytes = DkvSmem::total + 1024;

struct DkvParams {
  CUtensorMap map_k, map_v, map_q, map_dout, map_bias_t;
  oops_ta_pair dk, dv;
  const float* lse;
  const float* delta;
  const uint8_t* mask;
  int64_t m_sb, m_sr, m_sc;
  int batch, rows, cols, heads, bias_groups;
  int k_pairs, q_steps;
  int write_dk, write_dv;
  float scale;
};

template <typename T, bool HAS_BIAS>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) ta_bwd_dkv_kernel(const __grid_constant__ DkvParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + DkvSmem::abort_flag);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + DkvSmem::tmem_slot);
  auto bar = [&](int index) -> uint32_t { return smem_base + DkvSmem::bars + index * 8; };

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (device_failed()) return;
  int idx = blockIdx.x;
  const int kp = idx % P.k_pairs;
  idx /= P.k_pairs;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int r = idx % P.rows;
  const int b = idx / P.rows;
  const int k0 = kp * kTilesPerCta * kTile;
  const int n_tiles = (kTilesPerCta == 2 && k0 + kTile < P.cols) ? 2 : 1;
  const int QS = P.q_steps;
  const int g = P.bias_groups == 1 ? 0 : r;
  // tensor-memory columns of key tile w: S^T [0,64) | dP^T [64,128) | P^T [128,160) | dS^T [160,192) | dK [192,224) | dV [224,256)
  constexpr int kTileCols = 256, kDpCol = 64, kPCol = 128, kDsCol = 160, kDkCol = 192, kDvCol = 224;
  constexpr int kTmemCols = kTilesPerCta * kTileCols;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kTilesPerCta; ++i) {
      mbar_init(bar(DkvSmem::kv_full + i), 1);
      mbar_init(bar(DkvSmem::sd_full + i), 1);
      mbar_init(bar(DkvSmem::sd_free + i), 8);
      mbar_init(bar(DkvSmem::pds_full + i), 8);
      mbar_init(bar(DkvSmem::pds_done + i), 1);
      mbar_init(bar(DkvSmem::done + i), 1);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(bar(DkvSmem::qd_full + i), 1);
      mbar_init(bar(DkvSmem::qd_empty + i), 1);
    }
    for (int i = 0; i < 2 * kTilesPerCta; ++i) {
      mbar_init(bar(DkvSmem::bias_full + i), 1);
      mbar_init(bar(DkvSmem::bias_empty + i), 8);
    }
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_base + DkvSmem::tmem_slot, kTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kProducerWarp) {
    if (lane == 0) {
      bool ok = true;
      for (int w = 0; w < n_tiles; ++w) {
        mbar_expect_tx(bar(DkvSmem::kv_full + w), 2 * kBigTile);
        tma_load_5d(smem_base + DkvSmem::k + w * kBigTile, &P.map_k, bar(DkvSmem::kv_full + w), 0, h, k0 + w * kTile, r, b);
        tma_load_5d(smem_base + DkvSmem::v + w * kBigTile, &P.map_v, bar(DkvSmem::kv_full + w), 0, h, k0 + w * kTile, r, b);
      }
      for (int j = 0; j < QS && ok; ++j) {
        const int st = j % kRing, round = j / kRing;
        if (j >= kRing) ok = mbar_wait(bar(DkvSmem::qd_empty + st), (round - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(DkvSmem::qd_full + st), 2 * kSmallTile);
        const uint32_t dst = smem_base + DkvSmem::qd + st * 2 * kSmallTile;
        tma_load_5d(dst, &P.map_q, bar(DkvSmem::qd_full + st), 0, h, j * kStep, r, b);
        tma_load_5d(dst + kSmallTile, &P.map_dout, bar(DkvSmem::qd_full + st), 0, h, j * kStep, r, b);
        if (HAS_BIAS) {
          for (int w = 0; w < n_tiles && ok; ++w) {
            const int slot = w * 2 + (j & 1);
            if (j >= 2) ok = mbar_wait(bar(DkvSmem::bias_empty + slot), ((j >> 1) - 1) & 1, abort_flag);
            if (!ok) break;
            mbar_expect_tx(bar(DkvSmem::bias_full + slot), kBiasStep);
            // transposed bias: inner axis = query, outer axis = key
            tma_load_5d(smem_base + DkvSmem::bias + slot * kBiasStep, &P.map_bias_t, bar(DkvSmem::bias_full + slot),
                        j * kStep, k0 + w * kTile, h, g, b);
          }
        }
      }
    }
  } else if (warp == kMmaWarp || (kTilesPerCta == 2 && warp == kAccWarp)) {
    // One tile per CTA: one thread issues everything in the order the events arrive (scores of step j+1 when the
    // warpgroups have read step j, dV and dK of step j when they have stored P and dS).  Two tiles per CTA: a second
    // thread issues the dV/dK products, so that neither kind of product waits behind the other tile's barrier.
    if (lane == 0) {
      constexpr uint32_t fmt = Half2<T>::kFormat;
      constexpr uint32_t idesc_s = instr_desc(fmt, 0, 0, kTile, kStep);
      constexpr uint32_t idesc_acc = instr_desc(fmt, 0, 1, kTile, kHeadDim);
      const bool do_scores = warp == kMmaWarp, do_acc = kTilesPerCta == 1 || warp == kAccWarp;
      bool ok = true;
      // S^T[128 k x 64 q] = K Q^T and dP^T = V dO^T of step j for key tile w
      auto issue_scores = [&](int j, int w) {
        // the bias tile of the step has landed before the scores are announced: the warpgroups do not wait for it
        if (HAS_BIAS && !mbar_wait(bar(DkvSmem::bias_full + w * 2 + (j & 1)), (j >> 1) & 1, abort_flag)) return;
        const uint32_t qd = smem_base + DkvSmem::qd + (j % kRing) * 2 * kSmallTile;
        const uint32_t st_t = tmem_base + w * kTileCols;
        const uint64_t kdesc = smem_desc(smem_base + DkvSmem::k + w * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t vdesc = smem_desc(smem_base + DkvSmem::v + w * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t qdesc = smem_desc(qd, 16, 512, kSwizzle64B);
        const uint64_t ddesc = smem_desc(qd + kSmallTile, 16, 512, kSwizzle64B);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(st_t, kdesc + uint64_t(kk * 2), qdesc + uint64_t(kk * 2), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(st_t + kDpCol, vdesc + uint64_t(kk * 2), ddesc + uint64_t(kk * 2), idesc_s, kk > 0 ? 1u : 0u);
        mma_commit(bar(DkvSmem::sd_full + w));
      };
      auto issue_acc = [&](int j, int w) {
        const int st = j % kRing;
        const uint32_t tile_t = tmem_base + w * kTileCols;
        const uint32_t qd = smem_base + DkvSmem::qd + st * 2 * kSmallTile;
        const uint64_t qdesc = smem_desc(qd, 16, 512, kSwizzle64B);                 // Q step, MN-major
        const uint64_t ddesc = smem_desc(qd + kSmallTile, 16, 512, kSwizzle64B);    // dO step, MN-major
#pragma unroll
        for (int kk = 0; kk < kStep / 16; ++kk)  // dV[128 k x 32] += P^T[128 k x 64 q] dO[64 q x 32]
          mma_ts(tile_t + kDvCol, tile_t + kPCol + kk * 8, ddesc + uint64_t(kk * (1024 >> 4)), idesc_acc,
                 (j > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kStep / 16; ++kk)  // dK[128 k x 32] += dS^T[128 k x 64 q] Q[64 q x 32]
          mma_ts(tile_t + kDkCol, tile_t + kDsCol + kk * 8, qdesc + uint64_t(kk * (1024 >> 4)), idesc_acc,
                 (j > 0 || kk > 0) ? 1u : 0u);
        mma_commit(bar(DkvSmem::pds_done + w));
        if (j == QS - 1) mma_commit(bar(DkvSmem::done + w));
        if (w == n_tiles - 1) mma_commit(bar(DkvSmem::qd_empty + st));
      };
      if (do_scores) {
        for (int w = 0; w < n_tiles && ok; ++w) ok = mbar_wait(bar(DkvSmem::kv_full + w), 0, abort_flag);
        if (ok) ok = mbar_wait(bar(DkvSmem::qd_full), 0, abort_flag);
        if (ok) {
          tc_fence_after_sync();
          for (int w = 0; w < n_tiles; ++w) issue_scores(0, w);
        }
      }
      for (int j = 0; j < QS && ok; ++j) {
        if (do_scores && j + 1 < QS) {
          ok = mbar_wait(bar(DkvSmem::qd_full + (j + 1) % kRing), ((j + 1) / kRing) & 1, abort_flag);
          for (int w = 0; w < n_tiles && ok; ++w) {
            ok = mbar_wait(bar(DkvSmem::sd_free + w), j & 1, abort_flag);
            if (!ok) break;
            tc_fence_after_sync();
            issue_scores(j + 1, w);
          }
        }
        if (do_acc && ok) {
          if (!do_scores) ok = mbar_wait(bar(DkvSmem::qd_full + j % kRing), (j / kRing) & 1, abort_flag);
          for (int w = 0; w < n_tiles && ok; ++w) {
            ok = mbar_wait(bar(DkvSmem::pds_full + w), j & 1, abort_flag);
            if (!ok) break;
            tc_fence_after_sync();
            issue_acc(j, w);
          }
        }
      }
    }
  } else if (warp < kElemWarps && (warp >> 3) < n_tiles) {
    const int w = warp >> 3;           // key tile
    const int half = (warp >> 2) & 1;  // which 32 of the step's 64 queries
    const int t = tid & (kTile - 1);
    const uint32_t lane_field = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tile_t = tmem_base + lane_field + w * kTileCols;
    const int key = k0 + w * kTile + t;
    bool keep = key < P.cols;
    if (keep && P.mask) keep = P.mask[b * P.m_sb + int64_t(r) * P.m_sr + int64_t(key) * P.m_sc] != 0;
    const float scale = P.scale;
    const f32x2 c2 = pack2(scale * kLog2e, scale * kLog2e), log2e2 = pack2(kLog2e, kLog2e);
    const int64_t stat_base = ((int64_t(b) * P.rows + r) * P.heads + h) * P.cols;
    bool ok = true;

    // Row statistics of the step's 32 queries of this warpgroup's half: every warp keeps its own copy in shared
    // memory (no cross-warp barrier): lane i fetches -lse*log2e and -delta of query i one step ahead.
    // The loaded words are not touched until the next step (any arithmetic on them here would wait for the load).
    auto fetch_stats = [&](int j, float& lse_raw, float& delta_raw) {
      lse_raw = INFINITY;
      delta_raw = 0.f;
      const int q = j * kStep + half * 32 + lane;
      if (j < QS && q < P.cols) {
        lse_raw = ldg_f32_here(P.lse + stat_base + q);
        delta_raw = ldg_f32_here(P.delta + stat_base + q);
      }
    };
    float nl_next, nd_next;
    fetch_stats(0, nl_next, nd_next);
    for (int j = 0; j < QS && ok; ++j) {
      float* stats = reinterpret_cast<float*>(smem_gen + DkvSmem::stats + (warp * 2 + (j & 1)) * 256);
      stats[lane] = -nl_next * kLog2e;
      stats[32 + lane] = -nd_next;
      fetch_stats(j + 1, nl_next, nd_next);
      __syncwarp();
      ok = mbar_wait(bar(DkvSmem::sd_full + w), j & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      const int slot = w * 2 + (j & 1);
      const uint8_t* bias_row = smem_gen + DkvSmem::bias + slot * kBiasStep + t * 128 + (((t & 7) ^ (half * 4)) << 4);
      uint32_t p_packed[16], ds_packed[16];
      // two rounds of 16 queries keep the live registers low; the score columns are released after the second load
#pragma unroll
      for (int round = 0; round < 2; ++round) {
        uint32_t sraw[16], draw[16];
        tmem_ld16(tile_t + half * 32 + round * 16, sraw);
        tmem_ld16(tile_t + kDpCol + half * 32 + round * 16, draw);
        tmem_wait_ld();
        tmem_loaded(sraw);
        tmem_loaded(draw);
        if (round == 1) {
          tc_fence_before_sync();
          mbar_arrive_warp(bar(DkvSmem::sd_free + w));
        }
        if (keep) {
#pragma unroll
          for (int i8 = 0; i8 < 2; ++i8) {
            const int c8 = round * 2 + i8;  // which group of 8 queries of this half
            const float4 n01 = *reinterpret_cast<const float4*>(stats + c8 * 8);
            const float4 n23 = *reinterpret_cast<const float4*>(stats + c8 * 8 + 4);
            const float4 d01 = *reinterpret_cast<const float4*>(stats + 32 + c8 * 8);
            const float4 d23 = *reinterpret_cast<const float4*>(stats + 32 + c8 * 8 + 4);
            const f32x2 nl2[4] = {pack2(n01.x, n01.y), pack2(n01.z, n01.w), pack2(n23.x, n23.y), pack2(n23.z, n23.w)};
            const f32x2 nd2[4] = {pack2(d01.x, d01.y), pack2(d01.z, d01.w), pack2(d23.x, d23.y), pack2(d23.z, d23.w)};
            f32x2 p2[4], ds2[4];
            score_grad8<T, HAS_BIAS>(sraw + i8 * 8, draw + i8 * 8, swizzled_chunk(bias_row, c8), c2, log2e2,
                                     nl2, nd2, p2, ds2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              p_packed[c8 * 4 + i] = pack16<T>(p2[i]);
              ds_packed[c8 * 4 + i] = pack16<T>(ds2[i]);
            }
          }
        } else {
          // a dropped (or out-of-range) key contributes nothing, whatever its row holds
#pragma unroll
          for (int i = 0; i < 8; ++i) p_packed[round * 8 + i] = ds_packed[round * 8 + i] = 0u;
        }
      }
      if (HAS_BIAS) mbar_arrive_warp(bar(DkvSmem::bias_empty + slot));
      if (j > 0) {
        ok = mbar_wait(bar(DkvSmem::pds_done + w), (j - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
      }
      tmem_st16(tile_t + kPCol + half * 16, p_packed);
      tmem_st16(tile_t + kDsCol + half * 16, ds_packed);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive_warp(bar(DkvSmem::pds_full + w));
    }

    if (ok) ok = mbar_wait(bar(DkvSmem::done + w), 0, abort_flag);
    if (ok) {
      tc_fence_after_sync();
      uint32_t acc[32];
      if (half == 0 && P.write_dk) {
        tmem_ld32(tile_t + kDkCol, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
        if (key < P.cols) {
          T* dst = reinterpret_cast<T*>(P.dk.ptr) + b * P.dk.sb + int64_t(r) * P.dk.sr + int64_t(key) * P.dk.sc + h * P.dk.sh;
          store_row32<T>(dst, acc, scale, pair_vec_ok(P.dk));
        }
      }
      if (half == 1 && P.write_dv) {
        tmem_ld32(tile_t + kDvCol, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
        if (key < P.cols) {
          T* dst = reinterpret_cast<T*>(P.dv.ptr) + b * P.dv.sb + int64_t(r) * P.dv.sr + int64_t(key) * P.dv.sc + h * P.dv.sh;
          store_row32<T>(dst, acc, 1.f, pair_vec_ok(P.dv));
        }
      }
    }
  }
  teardown(abort_flag, tmem_base, kMmaWarp, kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// fused dQ / dK / dV kernel: one pass over the score tiles of a pair row
// ---------------------------------------------------------------------------------------------
// An item of the walk is a (batch, row, head).  Its query tiles are taken in groups of up to 6; for every group, every key
// tile and every query tile of the group: S = Q K^T and dP = dO V^T (128 x 128, tensor memory) -> the four warpgroups (a thread
// owns a query, a warpgroup 32 of the 128 keys) compute P and dS once and write them, 16-bit, into two shared-memory
// images whose rows are queries and whose 128-byte-swizzled columns are keys.  The tensor core reads those images three
// ways: dV += P^T dO and dK += dS^T Q take them as MN-major A operands (M = keys), dQ += dS K as a K-major A operand
// (M = queries).  dQ of the group's query tiles, dK and dV of the current key tile stay in tensor memory:
// S 128 | dP 128 | dK 32 | dV 32 | dQ 6 x 32 = 512 columns.  One `ex2` per logit and five products, where the
// separate dQ and dK/dV kernels spend two and seven.
// What bounds it: a step of some 2600 clocks spends 1100 in its arithmetic, where the exponentials (1024 clocks of the
// special-function units) and the issue slots are both full, and the rest in moving images, bias and scores (some 2000 clocks
// of the shared-memory port are busy) between barriers that all sixteen warps pass together.  Hence no branch, fence or
// generic-address store in a step's body, and the writers of the images do not fence: they release a barrier, and the
// issuer that acquires it fences once for all of them before its products read (N = 768: 1190 -> 1120 us with both).
// A statistics warp of its own puts -log2(e) lse and -delta of a part's queries into a table, a tile at a time and a part ahead, where every
// thread used to fetch both for every step (N = 768: 1036 -> 1004 us, 1024: 2934 -> 2842, 2048: 22.7 -> 22.0 ms), and makes the row dots where
// that is hidden (kOwnDeltaCols).  Where all rows of a sample keep the same first keys (closes_bias) the bias is minus infinity behind
// those, key tiles behind them are not walked, the statistics warp clears dropped keys and values in shared memory before any product may
// read them, and the element-wise warps know of no mask.  The launch that closes the bias looks at the mask first, and copies no sample that no
// walk needs closed (an all-ones mask of 768 columns: 5.0 -> 3.7 us, 2048: 20.8 -> 14.8).  Through other masks they test
// every probability, in a second copy of the step's body: a tile's way through the statistics warp, or bias words patched in
// registers instead, cost short rows 10 to 20 %.
// Halving the step between two sets of warps that run half a step apart was tried: the single P image couples them, 3 to 10 %
// slower.
// Rows of more than 768 columns have several groups.  The CTA walks them in order and carries the f32 sums of dK and
// dV of every key tile from group to group in a scratch slot that belongs to its SM (one CTA is resident per SM, so
// the slot is private while the CTA runs, and at 128 bytes per key and tensor it stays in L2): the thread that owns a
// key adds what the slot holds, and stores 16-bit dK/dV after the last group.  The order of the sums is fixed, so the
// gradients are bitwise reproducible, and no partial planes or reduction kernels exist.
// Where a row is one group, the CTA goes through several items without a stop: the copies and score products of the next one
// run under the last steps and the read-out of this one.  (A CTA per item spent half of its time on set-up and read-out at
// 256 columns: 4 steps in 26000 clocks.  N = 256: 86 -> 58 us, N = 768: 1190 -> 1032 us with what is named above.)

constexpr int kFMaxCols = 4096;          // longest row taken: 32 key tiles
constexpr int kFMaxQTiles = 6;
constexpr int kFThreads = 640;  // 16 element-wise warps, TMA producer, score issuer, accumulation issuer, statistics
constexpr int kFProducerWarp = 16, kFScoreWarp = 17, kFAccWarp = 18, kFStatWarp = 19;
constexpr int kFImage = 2 * 16384;       // P or dS of a step: two 64-key halves of 128 rows x 128 bytes
constexpr int kFBias = 2 * kBiasStep;    // 128 x 128 bias tile as two 64-key boxes (staging: copied to registers at once)
constexpr int kFSlots = 256;             // scratch slots of the group-to-group sums: one per SM id

struct FSmem {
  static constexpr int q = 0;                          // [3] 128 x 32 (a slot is held until the step's dK product ends)
  static constexpr int dout = q + 3 * kBigTile;        // [3]
  static constexpr int k = dout + 3 * kBigTile;        // [2]
  static constexpr int v = k + 2 * kBigTile;           // [2]
  static constexpr int ps = v + 2 * kBigTile;          // P image (read by the dV products only, freed early)
  static constexpr int dss = ps + kFImage;             // [2] dS image
  static constexpr int bias = dss + 2 * kFImage;       // one staging tile
  static constexpr int stats = bias + kFBias;          // [2][6][128] of two f32: statistics of a part's queries
  static constexpr int bars = stats + 2 * kFMaxQTiles * kTile * 8;
  static constexpr int qd_full = 0;                    // [3]
  static constexpr int qd_empty = qd_full + 3;         // [3]
  static constexpr int kv_full = qd_empty + 3;         // [2]
  static constexpr int kv_empty = kv_full + 2;         // [2]
  static constexpr int bias_full = kv_empty + 2;
  static constexpr int bias_empty = bias_full + 1;     // every warp has copied its words of the tile to registers
  static constexpr int sd_full = bias_empty + 1;       // S and dP of a step are in tensor memory
  static constexpr int sd_free = sd_full + 1;          // all warps have read them
  static constexpr int pds_full = sd_free + 1;         // [2] the P and dS images of a buffer are written
  static constexpr int pds_done = pds_full + 2;        // [2] the dK and dQ products have consumed the dS image
  static constexpr int p_done = pds_done + 2;          // the dV products have consumed the P image
  static constexpr int dkv_free = p_done + 1;          // dK and dV of a finished key tile have been read out
  static constexpr int dq_free = dkv_free + 1;         // dQ of a finished group of query tiles has been read out
  static constexpr int stat_full = dq_free + 1;        // [2][6] the statistics of a query tile stand
  static constexpr int stat_free = stat_full + 2 * kFMaxQTiles;  // [2] every warp is done with those of a part
  static constexpr int kv_ready = stat_free + 2;       // [2] dropped keys have been cleared (PREFIX)
  static constexpr int num_bars = kv_ready + 2;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int suspects = abort_flag + 4;      // query tiles with a row without a probability, perhaps
  static constexpr int total = suspects + 4;
};
constexpr int kFSmemBytes = FSmem::total + 1024;
static_assert(kFSmemBytes <= 232448, "fused reverse kernel: shared memory over the per-CTA limit");

struct FParams {
  CUtensorMap map_q, map_dout, map_k, map_v, map_bias, map_closed;
  oops_ta_pair dq, dk, dv;
  float* slots;     // [kFSlots][2][8][slot_keys][4] f32: sums of dK and dV carried from group to group (groups > 1)
  int64_t slot_keys;
  const float* lse;
  float* delta;     // read, or written from `out` and `dout` where own_delta is set
  oops_ta_pair out, dout;
  int own_delta;
  Logits logits;  // operands of a closed bias
  const uint8_t* mask;
  const uint32_t* live;  // what prepare_kernel has found out about the mask
  int64_t m_sb, m_sr, m_sc;
  int batch, rows, cols, heads, bias_groups, items;
  int q_tiles, k_tiles, groups, tiles_per_group;
  int write_dq, write_dk, write_dv;
  int closed;  // map_closed: the bias, minus infinity behind a ragged row's end or a token mask's, for walks without tests
  const uint32_t *prefix, *uniform;  // kept first keys of every row and of every sample's rows, null where nobody has looked
  float scale;
};

// Zeros for an item's rows from `first` on, by `threads` threads of which this is number `at`.
template <typename T>
__device__ __forceinline__ void store_zeros(const oops_ta_pair& t, const FParams& P, int item, int first, int at, int threads) {
  const int row = item / P.heads, b = row / P.rows;
  T* to = reinterpret_cast<T*>(t.ptr) + b * t.sb + int64_t(row - b * P.rows) * t.sr + int64_t(item - row * P.heads) * t.sh;
  const bool words = pair_vec_ok(t);
  for (int i = first * 4 + at; i < P.cols * 4; i += threads) {
    T* dst = to + int64_t(i >> 2) * t.sc + (i & 3) * 8;
    if (words) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    } else {
      for (int c = 0; c < 8; ++c) dst[c] = T(0.f);
    }
  }
}

// The walk over a CTA's steps, identical in every role of the kernel: parts outermost, then key tiles, then query tiles.
// A part is a group of query tiles of the CTA's one item, or, where a row is a single group, a whole item of the several
// that the CTA works through.  Ring slots and barrier phases count steps, key tiles and parts.  (Trip counts come from the
// launch parameters: with counts read from memory the compiler takes the loops for divergent and guards every
// branch in them, which cost the kernel 8 %.  The key tiles of a token mask are the exception: they come from memory once per CTA, through a shuffle
// that makes them one value for the warp, and without a loop over lanes before it.)
template <bool GROUPS>
struct FWalk {
  int tiles_per_group, q_tiles, k_tiles, parts, item_step;
  int part, item, first;  // part, its item, its first query tile
  int kt, qi, nq;         // key tile, query tile within the part, query tiles of the part
  int s, ktc;             // steps and key tiles walked so far
  __device__ FWalk(const FParams& P, int k_tiles)
      : tiles_per_group(P.tiles_per_group), q_tiles(P.q_tiles), k_tiles(k_tiles), parts(GROUPS ? P.groups : P.items),
        item_step(int(gridDim.x)), part(0), item(int(blockIdx.x)), first(0), kt(0), qi(0), nq(min(P.tiles_per_group, P.q_tiles)),
        s(0), ktc(0) {}
  __device__ bool done() const { return GROUPS ? part >= parts : item >= parts; }
  __device__ int qt() const { return GROUPS ? first + qi : qi; }
  __device__ void next_tile() {
    ++ktc;
    if (++kt < k_tiles) return;
    kt = 0;
    ++part;
    if (GROUPS) {
      first += tiles_per_group;
      nq = min(tiles_per_group, q_tiles - first);
    } else {
      item += item_step;
    }
  }
  __device__ void next() {
    ++s;
    if (++qi < nq) return;
    qi = 0;
    next_tile();
  }
};

// GROUPS: rows of several groups of query tiles.  BITS: some key may be dropped, by the mask or because the last key tile
// is ragged, and every probability is tested.  PREFIX: rows keep the first keys of their sample's prefix, or none, in `k_tiles` key tiles; dropped
// keys are cleared before a product reads them.  DIRECT: rows of one tile (below).
template <typename T, bool HAS_BIAS, bool GROUPS, bool BITS, bool PREFIX, bool DIRECT>
__device__ __forceinline__ void fused_walk(const FParams& P, uint32_t smem_base, uint8_t* smem_gen, volatile int* abort_flag,
                                           uint32_t tmem_base, int tid, int warp, int lane, int k_tiles) {
  auto bar = [&](int index) -> uint32_t { return smem_base + FSmem::bars + index * 8; };
  const bool has_mask = BITS && P.mask != nullptr;
  static_assert(!PREFIX || !BITS);
  auto request_prefix = [&](int item) -> uint32_t {  // every lane's copy; an item ahead of its use
    return PREFIX && item < P.items ? *reinterpret_cast<const volatile uint32_t*>(P.prefix + item / P.heads) : 0u;
  };
  // tensor-memory columns
  constexpr int kSCol = 0, kDpCol = 128, kDkCol = 256, kDvCol = 288, kDqCol = 320;

  if (warp == kFProducerWarp) {
    if (lane == 0) {
      bool ok = true;
      const CUtensorMap* map_bias = PREFIX || (P.closed && P.cols % kTile != 0) ? &P.map_closed : &P.map_bias;
      for (FWalk<GROUPS> w(P, k_tiles); !w.done() && ok; w.next()) {
        const int s = w.s, kt = w.kt, qt = w.qt(), qs = s % 3;
        const int row = w.item / P.heads, h = w.item - row * P.heads, b = row / P.rows, r = row - b * P.rows;
        if (w.qi == 0) {
          const int ks = w.ktc & 1;
          if (w.ktc >= 2) ok = mbar_wait(bar(FSmem::kv_empty + ks), ((w.ktc >> 1) - 1) & 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(FSmem::kv_full + ks), 2 * kBigTile);
          tma_load_5d(smem_base + FSmem::k + ks * kBigTile, &P.map_k, bar(FSmem::kv_full + ks), 0, h, kt * kTile, r, b);
          tma_load_5d(smem_base + FSmem::v + ks * kBigTile, &P.map_v, bar(FSmem::kv_full + ks), 0, h, kt * kTile, r, b);
        }
        if (s >= 3) ok = mbar_wait(bar(FSmem::qd_empty + qs), ((s / 3) - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(FSmem::qd_full + qs), 2 * kBigTile);
        tma_load_5d(smem_base + FSmem::q + qs * kBigTile, &P.map_q, bar(FSmem::qd_full + qs), 0, h, qt * kTile, r, b);
        tma_load_5d(smem_base + FSmem::dout + qs * kBigTile, &P.map_dout, bar(FSmem::qd_full + qs), 0, h, qt * kTile, r, b);
        if (HAS_BIAS) {
          if (s >= 1) ok = mbar_wait(bar(FSmem::bias_empty), (s - 1) & 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(FSmem::bias_full), kFBias);
          for (int box = 0; box < 2; ++box)
            tma_load_5d(smem_base + FSmem::bias + box * kBiasStep, map_bias, bar(FSmem::bias_full), kt * kTile + box * 64,
                        qt * kTile, h, P.bias_groups == 1 ? 0 : r, b);
        }
      }
    }
  } else if (warp == kFScoreWarp) {
    {
      constexpr uint32_t idesc = instr_desc(Half2<T>::kFormat, 0, 0, kTile, kTile);
      bool ok = true;
      for (FWalk<GROUPS> w(P, k_tiles); !w.done() && ok; w.next()) {
        const int s = w.s, qs = s % 3, ks = w.ktc & 1;
        ok = mbar_wait_warp(bar(FSmem::qd_full + qs), (s / 3) & 1, abort_flag);
        if (ok && w.qi == 0) ok = mbar_wait_warp(bar((PREFIX ? FSmem::kv_ready : FSmem::kv_full) + ks), (w.ktc >> 1) & 1, abort_flag);
        if (ok && s > 0) ok = mbar_wait_warp(bar(FSmem::sd_free), (s - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t qdesc = smem_desc(smem_base + FSmem::q + qs * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t ddesc = smem_desc(smem_base + FSmem::dout + qs * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t kdesc = smem_desc(smem_base + FSmem::k + ks * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t vdesc = smem_desc(smem_base + FSmem::v + ks * kBigTile, 16, 512, kSwizzle64B);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss_warp(tmem_base + kSCol, qdesc + uint64_t(kk * 2), kdesc + uint64_t(kk * 2), idesc, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss_warp(tmem_base + kDpCol, ddesc + uint64_t(kk * 2), vdesc + uint64_t(kk * 2), idesc, kk > 0 ? 1u : 0u);
        mma_commit_warp(bar(FSmem::sd_full));
      }
    }
  } else if (warp == kFAccWarp) {
    {
      constexpr uint32_t fmt = Half2<T>::kFormat;
      constexpr uint32_t idesc_t = instr_desc(fmt, 1, 1, kTile, kHeadDim);  // A = image^T (M = keys), B MN-major
      constexpr uint32_t idesc_q = instr_desc(fmt, 0, 1, kTile, kHeadDim);  // A = image (M = queries), B MN-major
      bool ok = true;
      for (FWalk<GROUPS> w(P, k_tiles); !w.done() && ok; w.next()) {
        const int s = w.s, kt = w.kt, qi = w.qi, qs = s % 3, ks = w.ktc & 1;
        ok = mbar_wait_warp(bar(FSmem::qd_full + qs), (s / 3) & 1, abort_flag);
        if (ok) ok = mbar_wait_warp(bar(FSmem::kv_full + ks), (w.ktc >> 1) & 1, abort_flag);
        if (ok) ok = mbar_wait_warp(bar(FSmem::pds_full + (s & 1)), (s >> 1) & 1, abort_flag);
        // dK and dV of the previous key tile must have been read out before they are overwritten,
        // and so must dQ of the previous part
        if (ok && qi == 0 && w.ktc > 0) ok = mbar_wait_warp(bar(FSmem::dkv_free), (w.ktc - 1) & 1, abort_flag);
        if (ok && qi == 0 && kt == 0 && w.part > 0) ok = mbar_wait_warp(bar(FSmem::dq_free), (w.part - 1) & 1, abort_flag);
        if (!ok) break;
        fence_proxy_async_smem();  // the images (and cleared key rows) were written through the generic proxy
        tc_fence_after_sync();
        const uint32_t ps = smem_base + FSmem::ps, dss = smem_base + FSmem::dss + (s & 1) * kFImage;
        const uint64_t qdesc = smem_desc(smem_base + FSmem::q + qs * kBigTile, 16, 512, kSwizzle64B);     // MN-major B
        const uint64_t ddesc = smem_desc(smem_base + FSmem::dout + qs * kBigTile, 16, 512, kSwizzle64B);  // MN-major B
        const uint64_t kdesc = smem_desc(smem_base + FSmem::k + ks * kBigTile, 16, 512, kSwizzle64B);       // MN-major B
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk)  // dV[128 k x 32] += P^T[128 k x 128 q] dO[128 q x 32]
          mma_ss_warp(tmem_base + kDvCol, smem_desc(ps + kk * 2048, 16384, 1024, kSwizzle128B), ddesc + uint64_t(kk * (1024 >> 4)),
                 idesc_t, (qi > 0 || kk > 0) ? 1u : 0u);
        mma_commit_warp(bar(FSmem::p_done));
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk)  // dK[128 k x 32] += dS^T[128 k x 128 q] Q[128 q x 32]
          mma_ss_warp(tmem_base + kDkCol, smem_desc(dss + kk * 2048, 16384, 1024, kSwizzle128B), qdesc + uint64_t(kk * (1024 >> 4)),
                 idesc_t, (qi > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk)  // dQ[128 q x 32] += dS[128 q x 128 k] K[128 k x 32]
          mma_ss_warp(tmem_base + kDqCol + qi * kHeadDim, smem_desc(dss + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024, kSwizzle128B),
                 kdesc + uint64_t(kk * (1024 >> 4)), idesc_q, (kt > 0 || kk > 0) ? 1u : 0u);
        mma_commit_warp(bar(FSmem::pds_done + (s & 1)));
        mma_commit_warp(bar(FSmem::qd_empty + qs));
        if (qi == w.nq - 1) mma_commit_warp(bar(FSmem::kv_empty + ks));
      }
    }
  } else if (warp == kFStatWarp && !DIRECT) {
    // Statistics of a part's queries, a tile at a time and a part ahead: -log2(e) lse, and -delta, which is rowsum(O * dO) where the
    // caller has not left it.  Four lanes share a query, eight channels each.
    bool ok = true;
    // Query tiles with a row that has no probability, perhaps (the forward pass leaves such a row a log-sum-exp of 0): looked at behind the walk.
    uint32_t suspects = 0;
    // `dead`: no key is kept, every probability, and dS, is zero.  `in_use`: the table holds a part that has to be through first (the words are
    // under way meanwhile).
    auto tile_stats = [&](int part, int item, int first, int qi, bool dead, bool in_use) {
      auto table_free = [&]() {
        if (in_use) ok = mbar_wait_warp(bar(FSmem::stat_free + (part & 1)), ((part >> 1) - 1) & 1, abort_flag);
        return ok;
      };
      const int buffer = part & 1, row = item / P.heads, h = item - row * P.heads, b = row / P.rows, r = row - b * P.rows;
      const int64_t stat = int64_t(item) * P.cols;
      const uint32_t table = smem_base + FSmem::stats + (buffer * kFMaxQTiles + qi) * (kTile * 8);
      const int q0 = (first + qi) * kTile;
      if (!P.own_delta) {
        float lse[4], delta[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int q = q0 + j * 32 + lane;
          lse[j] = q < P.cols ? ldg_f32_here(P.lse + stat + q) : INFINITY;
          delta[j] = q < P.cols ? ldg_f32_here(P.delta + stat + q) : 0.f;
        }
        if (!table_free()) return;
#pragma unroll
        for (int j = 0; j < 4; ++j) suspects |= lse[j] == 0.f && !dead ? 1u << (first + qi) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) sts_f2_at(table + (j * 32 + lane) * 8, dead ? -INFINITY : -lse[j] * kLog2e, dead ? 0.f : -delta[j]);
      } else {
        if (!table_free()) return;
        const T* po = reinterpret_cast<const T*>(P.out.ptr) + b * P.out.sb + int64_t(r) * P.out.sr + h * P.out.sh + (lane & 3) * 8;
        const T* pd = reinterpret_cast<const T*>(P.dout.ptr) + b * P.dout.sb + int64_t(r) * P.dout.sr + h * P.dout.sh + (lane & 3) * 8;
#pragma unroll 1
        for (int j = 0; j < kTile; j += 32) {
          const int q = q0 + j + lane;
          const float lse = q < P.cols ? ldg_f32_here(P.lse + stat + q) : INFINITY;
          uint4 o[4], g[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int at = q0 + j + i * 8 + (lane >> 2);
            o[i] = ldg_v4_here_if(po + int64_t(at) * P.out.sc, at < P.cols);
            g[i] = ldg_v4_here_if(pd + int64_t(at) * P.dout.sc, at < P.cols);
          }
          float own = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t ow[4] = {o[i].x, o[i].y, o[i].z, o[i].w}, gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
            float dot = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) dot += Half2<T>::lo(ow[e]) * Half2<T>::lo(gw[e]) + Half2<T>::hi(ow[e]) * Half2<T>::hi(gw[e]);
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
            const float mine = __shfl_sync(0xffffffffu, dot, (lane & 7) * 4);  // query i * 8 + lane % 8
            if ((lane >> 3) == i) own = mine;
          }
          if (q < P.cols) P.delta[stat + q] = own;
          suspects |= lse == 0.f && !dead ? 1u << (first + qi) : 0u;
          sts_f2_at(table + (j + lane) * 8, dead ? -INFINITY : -lse * kLog2e, dead ? 0.f : -own);
        }
      }
      mbar_arrive_warp(bar(FSmem::stat_full + buffer * kFMaxQTiles + qi));
    };
    FWalk<GROUPS> w(P, k_tiles);
    auto clear_key = [&](int slot, int key) {
      const uint32_t at = slot * kBigTile + key * 64;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        sts_v4_at(smem_base + FSmem::k + at + c * 16, make_uint4(0, 0, 0, 0));
        sts_v4_at(smem_base + FSmem::v + at + c * 16, make_uint4(0, 0, 0, 0));
      }
    };
    uint32_t item_kept = 0, next_kept = request_prefix(int(blockIdx.x));
    auto last = w;  // the key tile before
    if (!w.done()) tile_stats(0, w.item, w.first, 0, PREFIX && __shfl_sync(0xffffffffu, next_kept, 0) == 0, false);
    for (; !w.done() && ok; last = w, w.next_tile()) {
      const int kt = w.kt;
      if (PREFIX && kt == 0) {
        item_kept = __shfl_sync(0xffffffffu, next_kept, 0);
        next_kept = request_prefix(GROUPS ? w.item : w.item + int(gridDim.x));
      }
      const int slot = w.ktc & 1;
      if (PREFIX) {
        // (Every tile passes here, with dropped keys or not: this warp is then neither a phase of a slot behind nor two ahead.)
        ok = mbar_wait_warp(bar(FSmem::kv_full + slot), (w.ktc >> 1) & 1, abort_flag);
        if (!ok) break;
        if (item_kept < uint32_t(min(P.cols, (kt + 1) * kTile))) {
          for (int key = lane; key < kTile; key += 32)
            if (kt * kTile + key >= int(item_kept)) clear_key(slot, key);
          fence_proxy_async_smem();
        }
        mbar_arrive_warp(bar(FSmem::kv_ready + slot));
        if (!GROUPS && kt == k_tiles - 1) {  // what the element-wise warps leave out of the item
          if (P.write_dk) store_zeros<T>(P.dk, P, w.item, int(item_kept), lane, 32);
          if (P.write_dv) store_zeros<T>(P.dv, P, w.item, int(item_kept), lane, 32);
          if (P.write_dq && item_kept == 0) store_zeros<T>(P.dq, P, w.item, 0, lane, 32);
        }
      }
      // The query tiles of the first part, then one of the next part for every key tile of this one (the rest by the last, where keys have
      // fewer tiles): a key tile late, so that a tile with dropped keys does not wait for the table to be free.
      auto ahead = last;
      int from = 1, to = w.nq;
      if (w.ktc > 0) {
        ahead.kt = k_tiles - 1;
        ahead.next_tile();
        if (ahead.done()) continue;
        from = last.kt;
        to = last.kt == k_tiles - 1 ? ahead.nq : min(last.kt + 1, ahead.nq);
      }
      const bool dead = PREFIX && __shfl_sync(0xffffffffu, ahead.part == w.part ? item_kept : next_kept, 0) == 0;
#pragma unroll 1
      for (int qi = from; qi < to && ok; ++qi) tile_stats(ahead.part, ahead.item, ahead.first, qi, dead, qi == 0 && ahead.part >= 2);
    }
    if (HAS_BIAS && !BITS) {  // (tests drop what is dropped)
      suspects = __reduce_or_sync(0xffffffffu, suspects);
      if (lane == 0) *reinterpret_cast<volatile uint32_t*>(smem_gen + FSmem::suspects) = suspects;
    }
  } else if (warp < 16) {
    const int wg = warp >> 2;  // 32 of the step's 128 keys
    const int t = tid & (kTile - 1);
    const uint32_t lane_field = uint32_t((warp & 3) * 32) << 16;
    const uint32_t lanes_t = tmem_base + lane_field;
    const float scale = P.scale;
    const f32x2 c2 = pack2(scale * kLog2e, scale * kLog2e), log2e2 = pack2(kLog2e, kLog2e);
    // DIRECT: the statistics of this thread's query in a step's query tile, fetched one step ahead and left untouched till then.
    auto fetch_stats = [&](const FWalk<GROUPS>& at, float& lse_raw, float& delta_raw) {
      lse_raw = INFINITY;
      delta_raw = 0.f;
      const int q = at.qt() * kTile + t;
      if (!at.done() && q < P.cols) {
        const int64_t stat = int64_t(at.item) * P.cols + q;
        lse_raw = ldg_f32_here(P.lse + stat);
        delta_raw = ldg_f32_here(P.delta + stat);
      }
    };
    // The kept bit of this lane's key of a key tile (32 keys of this warpgroup), fetched a key tile ahead.
    auto mask_row_of = [&](int item) -> const uint8_t* {
      const int row = item / P.heads, b = row / P.rows;
      return P.mask + b * P.m_sb + int64_t(row - b * P.rows) * P.m_sr;
    };
    auto fetch_keep = [&](const uint8_t* row, const FWalk<GROUPS>& at) -> uint32_t {
      const int key = at.kt * kTile + wg * 32 + lane;
      if (at.done() || key >= P.cols) return 0;
      return has_mask ? ldg_u8_here(row + int64_t(key) * P.m_sc) : 1u;
    };
    const int row0 = int(blockIdx.x) / P.heads, h0 = int(blockIdx.x) - row0 * P.heads, b0 = row0 / P.rows, r0 = row0 - b0 * P.rows;
    auto item_row = [&](const oops_ta_pair& t, int item) -> T* {
      if (GROUPS) return reinterpret_cast<T*>(t.ptr) + b0 * t.sb + int64_t(r0) * t.sr + h0 * t.sh;
      const int row = item / P.heads, b = row / P.rows;
      return reinterpret_cast<T*>(t.ptr) + b * t.sb + int64_t(row - b * P.rows) * t.sr + int64_t(item - row * P.heads) * t.sh;
    };
    uint32_t sm_id;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm_id));
    // Kept keys of the item that is read out (several groups: at the read-out of the slot).  Nothing is stored for dropped keys and rows that
    // keep none, whose products a query or upstream gradient that is not finite makes NaN: the statistics warp writes their zeros.
    uint32_t kept = GROUPS ? 0u : request_prefix(int(blockIdx.x));
    // dK (warpgroup 0) and dV (warpgroup 1) of key tile kt, complete for the query tiles of group g: lanes are keys.
    // With several groups the f32 sums travel from group to group through this SM's scratch slot (the same thread
    // owns a key in every group), and the last group stores the 16-bit result.
    auto store_key_tile = [&](int item, int g, int kt) {
      if (wg > 1) return;
      uint32_t acc[32];
      tmem_ld32(lanes_t + (wg == 0 ? kDkCol : kDvCol), acc);
      tmem_wait_ld();
      tmem_loaded(acc);
      tc_fence_before_sync();
      mbar_arrive_warp(bar(FSmem::dkv_free));
      const bool wanted = wg == 0 ? P.write_dk != 0 : P.write_dv != 0;
      const int key = kt * kTile + t;
      if (key >= (PREFIX && !GROUPS ? int(kept) : P.cols)) return;
      if (!wanted) return;
      if (GROUPS) {
        // plane i of the slot holds channels 4i .. 4i+3 of every key, so that a warp's 32 keys are 512 contiguous bytes
        float4* slot = reinterpret_cast<float4*>(P.slots) + (int64_t(sm_id) * 2 + wg) * 8 * P.slot_keys + key;
        if (g == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            slot[i * P.slot_keys] = make_float4(__uint_as_float(acc[4 * i]), __uint_as_float(acc[4 * i + 1]),
                                                __uint_as_float(acc[4 * i + 2]), __uint_as_float(acc[4 * i + 3]));
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            red_add_f4(slot + i * P.slot_keys, __uint_as_float(acc[4 * i]), __uint_as_float(acc[4 * i + 1]),
                       __uint_as_float(acc[4 * i + 2]), __uint_as_float(acc[4 * i + 3]));
        }
        return;
      }
      const oops_ta_pair& o = wg == 0 ? P.dk : P.dv;
      store_row32<T>(item_row(o, item) + int64_t(key) * o.sc, acc, wg == 0 ? scale : 1.f, pair_vec_ok(o));
    };
    // dQ of a part, whose query tiles start with `first` (tile qi is read out by warpgroup qi % 4; lanes are queries); every
    // warp then reports that the accumulators may be overwritten by the next part
    auto store_query_tiles = [&](int item, int first) {
      const int tiles = min(P.tiles_per_group, P.q_tiles - first);
      const bool dead = PREFIX && !GROUPS && kept == 0;
      for (int qi = wg; qi < tiles; qi += 4) {
        uint32_t acc[32];
        tmem_ld32(lanes_t + kDqCol + qi * kHeadDim, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
        const int q_index = (first + qi) * kTile + t;
        if (q_index < P.cols && P.write_dq && !dead)
          store_row32<T>(item_row(P.dq, item) + int64_t(q_index) * P.dq.sc, acc, scale, pair_vec_ok(P.dq));
      }
      tc_fence_before_sync();
      mbar_arrive_warp(bar(FSmem::dq_free));
    };
    FWalk<GROUPS> w(P, k_tiles);
    float lse_next = 0.f, delta_next = 0.f;
    if (DIRECT) fetch_stats(w, lse_next, delta_next);
    const uint8_t* mask_row = has_mask ? mask_row_of(w.item) : nullptr;  // of the key tile to come
    uint32_t keep_raw = BITS ? fetch_keep(mask_row, w) : 0u, bits = 0xffffffffu;
    bool ok = true;
    if (GROUPS && sm_id >= uint32_t(kFSlots)) {  // no scratch slot for this SM id: give up like a wait that ran out
      *abort_flag = 1;
      ok = false;
    }

    // bias row of this thread's query in the staging tile: box (wg >> 1), 16-byte chunks (wg & 1) * 4 .. + 3
    const uint8_t* bias_row = smem_gen + FSmem::bias + (wg >> 1) * kBiasStep + t * 128 + (((t & 7) ^ ((wg & 1) * 4)) << 4);

    int last_item = 0, last_part = 0, last_first = 0, last_kt = 0;  // of the previous step
    for (; !w.done() && ok; last_item = w.item, last_part = w.part, last_first = w.first, last_kt = w.kt, w.next()) {
      const int s = w.s, kt = w.kt, qi = w.qi, buf = s & 1, table = (w.part & 1) * kFMaxQTiles + qi;
      if (BITS && qi == 0) {
        bits = __ballot_sync(0xffffffffu, keep_raw != 0);
        FWalk<GROUPS> ahead = w;
        ahead.next_tile();
        if (!GROUPS && has_mask && ahead.kt == 0 && !ahead.done()) mask_row = mask_row_of(ahead.item);
        keep_raw = fetch_keep(mask_row, ahead);
        if (has_mask && bits != 0xffffffffu) {
          // Key rows of dropped keys must not reach the dQ product (0 * inf): they are cleared in shared memory, eight of
          // this warpgroup's 32 by each warp.  The scores of these keys are dropped whatever they are.
          ok = mbar_wait(bar(FSmem::kv_full + (w.ktc & 1)), (w.ktc >> 1) & 1, abort_flag);
          if (!ok) break;
          const int key = (warp & 3) * 8 + (lane >> 2);
          if (((bits >> key) & 1u) == 0)
            sts_v4_at(smem_base + FSmem::k + (w.ktc & 1) * kBigTile + (wg * 32 + key) * 64 + (lane & 3) * 16, make_uint4(0, 0, 0, 0));
        }
      }
      if (s > 0) mbar_arrive_warp(bar(FSmem::pds_full + (buf ^ 1)));  // the images of step s - 1, their stores drained by now
      // The three phases the step needs first are probed together (one round trip to the barrier words); in the steady
      // state, where these warps are the slow side of the pipeline, all three are complete.
      const bool bias_there = HAS_BIAS && mbar_test(bar(FSmem::bias_full), s & 1);
      const bool image_free = s < 2 || mbar_test(bar(FSmem::pds_done + buf), ((s >> 1) - 1) & 1);
      const bool scores_there = mbar_test(bar(FSmem::sd_full), s & 1);
      float neg_lse2, neg_delta;
      if (DIRECT) {
        neg_lse2 = -lse_next * kLog2e;
        neg_delta = -delta_next;
        FWalk<GROUPS> ahead = w;
        ahead.next();
        fetch_stats(ahead, lse_next, delta_next);
      } else {
        const bool stats_there = kt > 0 || mbar_test(bar(FSmem::stat_full + table), (w.part >> 1) & 1);
        ok = mbar_wait_probed(stats_there, bar(FSmem::stat_full + table), (w.part >> 1) & 1, abort_flag);
        if (!ok) break;
        lds_f2_at(smem_base + FSmem::stats + (table * kTile + t) * 8, neg_lse2, neg_delta);
      }
      const f32x2 nl1 = pack2(neg_lse2, neg_lse2), nd1 = pack2(neg_delta, neg_delta);
      // The step's bias words are requested at once; the staging tile is handed back as soon as they have arrived
      // (below, after the first scores have been fetched), so that the next tile's copy runs under this step's arithmetic.
      uint4 bias_words[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      if (HAS_BIAS) {
        ok = mbar_wait_probed(bias_there, bar(FSmem::bias_full), s & 1, abort_flag);
        if (!ok) break;
#pragma unroll
        for (int c = 0; c < 4; ++c) bias_words[c] = lds_v4_here(swizzled_chunk(bias_row, c));
      }
      // this step's dS image was last read by the products of step s - 2, the P image by the dV products of s - 1
      ok = mbar_wait_probed(image_free, bar(FSmem::pds_done + buf), ((s >> 1) - 1) & 1, abort_flag);
      if (ok) ok = mbar_wait_probed(scores_there, bar(FSmem::sd_full), s & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      // image rows are queries; this warpgroup's 32 keys are chunks (wg & 1) * 4 .. + 3 of half (wg >> 1)
      const int row_at = (wg >> 1) * 16384 + t * 128 + (((t & 7) ^ ((wg & 1) * 4)) << 4);
      const uint32_t p_row = smem_base + FSmem::ps + row_at;
      const uint32_t ds_row = smem_base + FSmem::dss + buf * kFImage + row_at;
      uint32_t p_packed[16];
      bool p_free = s < 1;
      // (Two copies of the body: a test per eight columns splits the step into blocks that the compiler cannot interleave.)
      auto step_body = [&](auto drops_keys) {
        // Eight columns of S and dP at a time; the next eight are requested as soon as the current ones have arrived
        // and travel under the current eight's arithmetic.
        uint32_t sraw[2][8], draw[2][8];
        tmem_ld8(lanes_t + kSCol + wg * 32, sraw[0]);
        tmem_ld8(lanes_t + kDpCol + wg * 32, draw[0]);
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {
          tmem_wait_ld();
          tmem_loaded(sraw[c8 & 1]);
          tmem_loaded(draw[c8 & 1]);
          if (c8 == 0 && HAS_BIAS) {
            // the bias words must have returned before the tile is handed back (the copy of the next tile may land at once)
#pragma unroll
            for (int c = 0; c < 4; ++c)
              asm volatile("" ::"r"(bias_words[c].x), "r"(bias_words[c].y), "r"(bias_words[c].z), "r"(bias_words[c].w) : "memory");
            mbar_arrive_warp(bar(FSmem::bias_empty));
          }
          if (c8 < 3) {
            tmem_ld8(lanes_t + kSCol + wg * 32 + (c8 + 1) * 8, sraw[(c8 + 1) & 1]);
            tmem_ld8(lanes_t + kDpCol + wg * 32 + (c8 + 1) * 8, draw[(c8 + 1) & 1]);
          } else {
            tc_fence_before_sync();
            mbar_arrive_warp(bar(FSmem::sd_free));
            // the P image's phase is probed here; the answer travels under the last eight columns' arithmetic
            if (s >= 1) p_free = mbar_test(bar(FSmem::p_done), (s - 1) & 1);
          }
          f32x2 p2[4], ds2[4];
          score_grad8_words<T, HAS_BIAS>(sraw[c8 & 1], draw[c8 & 1], bias_words[c8], c2, log2e2, nl1, nd1, p2, ds2);
          if (decltype(drops_keys)::value) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              p2[i] = select2(p2[i], bits, c8 * 8 + 2 * i);
              ds2[i] = select2(ds2[i], bits, c8 * 8 + 2 * i);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) p_packed[c8 * 4 + i] = pack16<T>(p2[i]);
          sts_v4_at(ds_row ^ uint32_t(c8 << 4),
                    make_uint4(pack16<T>(ds2[0]), pack16<T>(ds2[1]), pack16<T>(ds2[2]), pack16<T>(ds2[3])));
        }
      };
      if (bits == 0xffffffffu)
        step_body(std::false_type{});
      else
        step_body(std::true_type{});
      // the single P image is free once the dV products of the previous step have read it; by now they have
      ok = mbar_wait_probed(p_free, bar(FSmem::p_done), (s - 1) & 1, abort_flag);
      if (!ok) break;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        sts_v4_at(p_row ^ uint32_t(c << 4),
                  make_uint4(p_packed[4 * c], p_packed[4 * c + 1], p_packed[4 * c + 2], p_packed[4 * c + 3]));
      if (qi == 0 && s > 0) {
        // A new key tile: dK and dV of the previous one are complete once the products of step s - 1 are (a commit
        // covers every product issued before it); a new group also finds its predecessor's dQ complete.  The products
        // of step s, which overwrite these accumulators, are issued after this step's images have been handed over,
        // which happens at the top of the next step: they wait for the read-out through dkv_free / dq_free only.
        ok = mbar_wait(bar(FSmem::pds_done + ((s - 1) & 1)), ((s - 1) >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        store_key_tile(last_item, last_part, last_kt);
        if (kt == 0) {
          store_query_tiles(last_item, last_first);
          if (!GROUPS) kept = request_prefix(w.item);  // (it has a key tile's time to arrive)
          mbar_arrive_warp(bar(FSmem::stat_free + ((w.part & 1) ^ 1)));
        }
      }
    }
    const int steps = w.s;
    if (ok && steps > 0) {  // the images of the last step
      mbar_arrive_warp(bar(FSmem::pds_full + ((steps - 1) & 1)));
    }

    // every product has finished when the products of the last step have
    if (ok && steps > 0) ok = mbar_wait(bar(FSmem::pds_done + ((steps - 1) & 1)), ((steps - 1) >> 1) & 1, abort_flag);
    if (ok && steps > 0) {
      tc_fence_after_sync();
      store_key_tile(last_item, last_part, last_kt);
      store_query_tiles(last_item, last_first);
    }
    if (GROUPS) {
      // The row's dK and dV now stand complete in this SM's slot (f32, summed group by group in a fixed order by the
      // thread that owns the key).  Every warp passes the barrier, whatever became of its waits; the 16-bit rows are
      // then written by all of them: four lanes share a key, so a warp stores eight 64-byte rows per instruction.
      __threadfence();
      named_barrier_sync(2, 16 * 32);
      if (*abort_flag == 0) {
        const int words = 2 * P.cols * 4;  // (tensor, key, eight channels)
        const int ends = PREFIX ? int(request_prefix(int(blockIdx.x))) : P.cols;
        for (int at = tid; at < words; at += 16 * 32) {
          const int j = at & 3, key = (at >> 2) % P.cols, which = (at >> 2) / P.cols;
          const bool wanted = which == 0 ? P.write_dk != 0 : P.write_dv != 0;
          if (!wanted) continue;
          const float4* slot = reinterpret_cast<const float4*>(P.slots) + (int64_t(sm_id) * 2 + which) * 8 * P.slot_keys + key;
          float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
          if (!PREFIX || key < ends) {  // (behind the last key tile that is walked the slot holds what another row has left)
            lo = ldcg_f4(slot + (2 * j) * P.slot_keys);
            hi = ldcg_f4(slot + (2 * j + 1) * P.slot_keys);
          }
          const float f = which == 0 ? scale : 1.f;
          const oops_ta_pair& o = which == 0 ? P.dk : P.dv;
          T* dst = item_row(o, int(blockIdx.x)) + int64_t(key) * o.sc + j * 8;
          const uint32_t w0 = Half2<T>::pack(lo.x * f, lo.y * f), w1 = Half2<T>::pack(lo.z * f, lo.w * f);
          const uint32_t w2 = Half2<T>::pack(hi.x * f, hi.y * f), w3 = Half2<T>::pack(hi.z * f, hi.w * f);
          if (pair_vec_ok(o)) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(w0, w1, w2, w3);
          } else {
            unsigned short* d0 = reinterpret_cast<unsigned short*>(dst);
            const uint32_t ws[4] = {w0, w1, w2, w3};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              d0[2 * i] = (unsigned short)(ws[i] & 0xffffu);
              d0[2 * i + 1] = (unsigned short)(ws[i] >> 16);
            }
          }
        }
      }
    }
  }
}

// MASKED: there is a mask or a ragged last key tile.  A mask that keeps everything takes the walk without tests (the
// tests, and above all what they do to the compiler's schedule, cost 8 %).
// DIRECT: rows of one tile, whose statistics every thread fetches itself: one step of an item is too short to hide the way through the table
// (64 columns 11.8 -> 10.6 us).
template <typename T, bool HAS_BIAS, bool GROUPS, bool MASKED, bool DIRECT>
__global__ void __launch_bounds__(kFThreads, 1) ta_bwd_fused_kernel(const __grid_constant__ FParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + FSmem::abort_flag);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + FSmem::tmem_slot);
  auto bar = [&](int index) -> uint32_t { return smem_base + FSmem::bars + index * 8; };

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (device_failed()) return;
  if (warp == 0) {  // a lane each: one thread took half a microsecond for them
    for (int i = lane; i < FSmem::num_bars; i += 32) {
      int arrivals = 1;
      if (i == FSmem::bias_empty || i == FSmem::sd_free || i == FSmem::dq_free) arrivals = 16;
      if (i == FSmem::pds_full || i == FSmem::pds_full + 1 || i == FSmem::stat_free || i == FSmem::stat_free + 1) arrivals = 16;
      if (i == FSmem::dkv_free) arrivals = 8;
      mbar_init(bar(i), arrivals);
    }
    if (lane == 0) {
      *abort_flag = 0;
      *reinterpret_cast<volatile uint32_t*>(smem_gen + FSmem::suspects) = 0;
    }
    fence_barrier_init();
  }
  if (warp == kFScoreWarp) {
    tmem_alloc(smem_base + FSmem::tmem_slot, 512);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bool plain = !MASKED;
  if (MASKED && P.mask && (P.cols % kTile == 0 || P.closed)) plain = keeps_all(P.live, P.batch * P.rows, lane);
  if (plain) {
    fused_walk<T, HAS_BIAS, GROUPS, false, false, DIRECT>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, P.k_tiles);
  } else if constexpr (MASKED) {
    uint32_t most = 0;
    const bool uniform = HAS_BIAS && !DIRECT && P.uniform && uniform_prefix(P.uniform, P.batch, lane, most);
    if (GROUPS && uniform && *reinterpret_cast<const volatile uint32_t*>(P.prefix + blockIdx.x / uint32_t(P.heads)) == 0) {
      // The CTA's one row keeps no key: zeros.
      if (P.write_dq) store_zeros<T>(P.dq, P, int(blockIdx.x), 0, tid, kFThreads);
      if (P.write_dk) store_zeros<T>(P.dk, P, int(blockIdx.x), 0, tid, kFThreads);
      if (P.write_dv) store_zeros<T>(P.dv, P, int(blockIdx.x), 0, tid, kFThreads);
    } else if (uniform)
      fused_walk<T, HAS_BIAS, GROUPS, false, HAS_BIAS, false>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane,
                                                       __shfl_sync(0xffffffffu, max(1, int(most + kTile - 1) / kTile), 0));
    else
      fused_walk<T, HAS_BIAS, GROUPS, true, false, DIRECT>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, P.k_tiles);
  }
  teardown(abort_flag, tmem_base, kFScoreWarp);
  if (HAS_BIAS && !DIRECT && P.closed && P.write_dq) {
    // A query that holds an infinity has NaN for the zeros of keys that the bias closes.  A row whose kept logits are minus infinity, all of
    // them, has no probability and no gradient all the same; its dQ stands by now.  A warp takes 32 queries of an item.
    const uint32_t suspects = *reinterpret_cast<volatile uint32_t*>(smem_gen + FSmem::suspects);
    const int item_step = GROUPS ? P.items : int(gridDim.x), chunks = (P.cols + 31) / 32;
    int item = int(blockIdx.x);
    for (int at = warp; suspects != 0 && item < P.items; at += kFThreads / 32) {
      for (; at >= chunks && item < P.items; at -= chunks) item += item_step;
      const int q = at * 32 + lane;
      if (item >= P.items || (suspects >> (at / 4) & 1u) == 0 || q >= P.cols) continue;
      const int row = item / P.heads, h = item - row * P.heads, b = row / P.rows, r = row - b * P.rows;
      T* dq = reinterpret_cast<T*>(P.dq.ptr) + b * P.dq.sb + int64_t(r) * P.dq.sr + int64_t(q) * P.dq.sc + h * P.dq.sh;
      if (P.lse[int64_t(item) * P.cols + q] != 0.f || !isnan(float(*dq))) continue;
      const int kept = P.prefix && P.uniform[b] != ~0u ? int(P.prefix[row]) : P.cols;
      if (!P.logits.all_minus_infinity<T>(b, r, h, q, kept)) continue;
      for (int c = 0; c < kHeadDim; ++c) dq[c] = T(0.f);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// shared-bias gradient kernel
// ---------------------------------------------------------------------------------------------
// dBias[b, h, q, k] = sum over rows r of dS[b, r, h, q, k].  The sum runs over the rows, so this kernel's loop nest has
// the rows innermost: a CTA owns one 128-query x 128-key tile of one (batch, head) and walks the rows of its part.
// Per row the tensor core produces S = Q K^T and dP = dO V^T (two 128 x 128 x 32 products, full-rate N = 128
// instructions, double-buffered in all 512 tensor-memory columns) and the sixteen element-wise warps (a thread owns
// one query and 32 of the tile's keys) add dS into f32 registers.  Everything that does not depend on the row stays
// in registers for the whole kernel: the thread's 32 bias values, already multiplied by log2(e), and the running
// sums.  Per logit the loop then costs one packed add (bias - lse), one packed multiply-add (exponent), `ex2`, one
// packed add (dP - delta) and one packed multiply-add (sum += P (dP - delta)).  With enough tiles to fill the SMs there is a single part and the CTA stores
// the final 16-bit gradient itself; small problems split the rows into parts whose f32 planes a last kernel adds in a
// fixed order (no atomics, bitwise reproducible either way).

constexpr int kDbRing = 4;
constexpr int kDbListRows = 8192;       // longest part whose rows without a kept key are passed over
constexpr int kDbStage = 4 * kBigTile;  // Q | dO | K | V of one row: 128 x 32 each
struct DbSmem {
  static constexpr int bias = 0;                         // 128 queries x 128 keys as two 64-key boxes (prologue only)
  static constexpr int ring = bias + 2 * kBiasStep;      // [kDbRing] stages
  static constexpr int bars = ring + kDbRing * kDbStage;
  static constexpr int bias_full = 0;
  static constexpr int row_full = 1;                     // [kDbRing]
  static constexpr int row_empty = row_full + kDbRing;   // [kDbRing]
  static constexpr int sd_full = row_empty + kDbRing;    // [2]
  static constexpr int sd_free = sd_full + 2;            // [2]
  static constexpr int num_bars = sd_free + 2;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int row_count = abort_flag + 4;
  static constexpr int keys_end = row_count + 4;
  static constexpr int row_list = (keys_end + 4 + 15) / 16 * 16;  // [kDbListRows] u16: rows of the part with a kept key in the tile
  static constexpr int total = row_list + kDbListRows * 2;
};
constexpr int kDbSmemBytes = DbSmem::total + 1024;
static_assert(kDbSmemBytes <= 232448, "shared-bias kernel: shared memory over the per-CTA limit");

struct DbParams {
  CUtensorMap map_q, map_dout, map_k, map_v, map_bias;
  float* parts;  // [parts][batch][heads][cols][cols] f32 (num_parts > 1)
  void* dbias;   // final gradient (num_parts == 1): the bias type, or f32 when dbias_f32 is set
  int64_t db_sb, db_sh, db_sq, db_sk;
  int dbias_f32;
  const float* lse;
  const float* delta;
  const uint8_t* mask;
  const uint32_t* live;  // [batch][rows] key tiles with a kept key (with a mask and at most 32 key tiles)
  int64_t m_sb, m_sr, m_sc;
  int batch, rows, cols, heads;
  int tiles, num_parts, rows_per_part;
  float scale;
};

// BITS: rows may drop keys of the tile, each its own; otherwise they keep the same ones, those before `end`.  LISTED: the rows
// that keep no key of the tile add nothing, and every role walks the others through a list.
template <typename T, bool BITS, bool LISTED>
__device__ __forceinline__ void dbias_walk(const DbParams& P, uint32_t smem_base, uint8_t* smem_gen, volatile int* abort_flag,
                                           uint32_t tmem_base, int tid, int warp, int lane, int b, int h, int qt, int kt, int part,
                                           int row_lo, int part_rows, int end) {
  auto bar = [&](int index) -> uint32_t { return smem_base + DbSmem::bars + index * 8; };
  const bool has_mask = BITS && P.mask != nullptr;
  const uint16_t* row_list = reinterpret_cast<const uint16_t*>(smem_gen + DbSmem::row_list);
  const int n_rows = LISTED ? *reinterpret_cast<volatile int*>(smem_gen + DbSmem::row_count) : part_rows;
  auto part_row = [&](int i) -> int { return LISTED ? int(row_list[i]) : i; };  // i-th row walked, counted within the part

  if (warp == kDbProducerWarp) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(bar(DbSmem::bias_full), 2 * kBiasStep);
      for (int box = 0; box < 2; ++box)
        tma_load_5d(smem_base + DbSmem::bias + box * kBiasStep, &P.map_bias, bar(DbSmem::bias_full), kt * kTile + box * 64,
                    qt * kTile, h, 0, b);
      for (int i = 0; i < n_rows && ok; ++i) {
        const int st = i % kDbRing, round = i / kDbRing, r = row_lo + part_row(i);
        if (i >= kDbRing) ok = mbar_wait(bar(DbSmem::row_empty + st), (round - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(DbSmem::row_full + st), kDbStage);
        const uint32_t dst = smem_base + DbSmem::ring + st * kDbStage;
        tma_load_5d(dst, &P.map_q, bar(DbSmem::row_full + st), 0, h, qt * kTile, r, b);
        tma_load_5d(dst + kBigTile, &P.map_dout, bar(DbSmem::row_full + st), 0, h, qt * kTile, r, b);
        tma_load_5d(dst + 2 * kBigTile, &P.map_k, bar(DbSmem::row_full + st), 0, h, kt * kTile, r, b);
        tma_load_5d(dst + 3 * kBigTile, &P.map_v, bar(DbSmem::row_full + st), 0, h, kt * kTile, r, b);
      }
    }
  } else if (warp == kDbMmaWarp) {
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc(Half2<T>::kFormat, 0, 0, kTile, kTile);
      bool ok = true;
      for (int i = 0; i < n_rows && ok; ++i) {
        const int st = i % kDbRing, buf = i & 1;
        ok = mbar_wait(bar(DbSmem::row_full + st), (i / kDbRing) & 1, abort_flag);
        if (ok && i >= 2) ok = mbar_wait(bar(DbSmem::sd_free + buf), ((i >> 1) - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t base = smem_base + DbSmem::ring + st * kDbStage;
        const uint64_t qdesc = smem_desc(base, 16, 512, kSwizzle64B);
        const uint64_t ddesc = smem_desc(base + kBigTile, 16, 512, kSwizzle64B);
        const uint64_t kdesc = smem_desc(base + 2 * kBigTile, 16, 512, kSwizzle64B);
        const uint64_t vdesc = smem_desc(base + 3 * kBigTile, 16, 512, kSwizzle64B);
        const uint32_t s_t = tmem_base + buf * 2 * kTile;
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(s_t, qdesc + uint64_t(kk * 2), kdesc + uint64_t(kk * 2), idesc, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(s_t + kTile, ddesc + uint64_t(kk * 2), vdesc + uint64_t(kk * 2), idesc, kk > 0 ? 1u : 0u);
        mma_commit(bar(DbSmem::sd_full + buf));
        mma_commit(bar(DbSmem::row_empty + st));
      }
    }
  } else if (warp < kDbElemWarps) {
    const int wg = warp >> 2;  // 32 of the tile's 128 keys
    const int t = tid & (kTile - 1);
    const uint32_t lane_field = uint32_t((warp & 3) * 32) << 16;
    const int q_index = qt * kTile + t;
    const bool q_valid = q_index < P.cols;
    const int key_base = kt * kTile + wg * 32;
    const float scale = P.scale;
    const f32x2 c2 = pack2(scale * kLog2e, scale * kLog2e);

    // The thread's bias values, times log2(e), for the whole kernel.
    bool ok = mbar_wait(bar(DbSmem::bias_full), 0, abort_flag);
    f32x2 bias2[16];
    {
      const uint8_t* bias_row = smem_gen + DbSmem::bias + (wg >> 1) * kBiasStep + t * 128 + (((t & 7) ^ ((wg & 1) * 4)) << 4);
      const f32x2 log2e2 = pack2(kLog2e, kLog2e);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (ok) v = *reinterpret_cast<const uint4*>(swizzled_chunk(bias_row, c));
        bias2[4 * c + 0] = mul2(Half2<T>::widen(v.x), log2e2);
        bias2[4 * c + 1] = mul2(Half2<T>::widen(v.y), log2e2);
        bias2[4 * c + 2] = mul2(Half2<T>::widen(v.z), log2e2);
        bias2[4 * c + 3] = mul2(Half2<T>::widen(v.w), log2e2);
      }
    }
    f32x2 acc2[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc2[i] = pack2(0.f, 0.f);

    const bool need_bits = BITS && (has_mask || key_base + 32 > P.cols);
    const int64_t stat_stride = int64_t(P.heads) * P.cols;
    const int64_t stat_first = ((int64_t(b) * P.rows + row_lo) * P.heads + h) * P.cols + q_index;
    // Prefetch of the next row's statistics and mask byte: the loaded words stay untouched until that row's turn
    // (any arithmetic on them here would wait for the load).
    int ahead = n_rows > 0 ? part_row(0) : 0;  // the row whose words are fetched next: list entries are read a row earlier still
    auto load_stats = [&](int i, float& lse_raw, float& delta_raw, uint32_t& keep_raw) {
      lse_raw = INFINITY;
      delta_raw = 0.f;
      keep_raw = 0;
      if (i < n_rows) {
        const int at = LISTED ? ahead : i, r = row_lo + at;
        if (q_valid) {
          lse_raw = ldg_f32_here(P.lse + stat_first + int64_t(at) * stat_stride);
          delta_raw = ldg_f32_here(P.delta + stat_first + int64_t(at) * stat_stride);
        }
        const int key = key_base + lane;
        if (key < P.cols) {
          keep_raw = 1;
          if (has_mask) keep_raw = ldg_u8_here(P.mask + b * P.m_sb + int64_t(r) * P.m_sr + int64_t(key) * P.m_sc);
        }
      }
    };
    float next_lse, next_dl;
    uint32_t next_keep;
    load_stats(0, next_lse, next_dl, next_keep);
    if (LISTED) ahead = row_list[1];

    bool scores_there = false;  // answer of the probe the previous row sent for this row's scores
    for (int i = 0; i < n_rows && ok; ++i) {
      const int buf = i & 1;
      const float neg_lse2 = -next_lse * kLog2e, neg_delta = -next_dl;
      const bool keep_lane = next_keep != 0;
      load_stats(i + 1, next_lse, next_dl, next_keep);
      if (LISTED) ahead = row_list[min(i + 2, kDbListRows - 1)];
      const uint32_t bits = need_bits ? __ballot_sync(0xffffffffu, keep_lane) : 0xffffffffu;
      const f32x2 nl1 = pack2(neg_lse2, neg_lse2), nd1 = pack2(neg_delta, neg_delta);
      ok = mbar_wait_probed(scores_there, bar(DbSmem::sd_full + buf), (i >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      scores_there = false;
      const uint32_t s_t = tmem_base + lane_field + buf * 2 * kTile + wg * 32;
      // The row's 32 logits of this thread, four tensor-memory columns of S and of dP at a time.  Rows with a dropped
      // key take a second copy of the body that zeroes the dropped columns: a test per element inside one body
      // would be compiled into selects that every row pays for.
      auto row_body = [&](auto drops_keys) {
        // two pairs (four tensor-memory columns of S and of dP) at a time; the loads of the next four columns are in
        // flight while the current four are worked on
        auto work4 = [&](int quad, const uint32_t (&sraw)[4], const uint32_t (&draw)[4]) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int pair = quad * 2 + j;
            const f32x2 s2 = pack2(__uint_as_float(sraw[2 * j]), __uint_as_float(sraw[2 * j + 1]));
            const f32x2 d2 = pack2(__uint_as_float(draw[2 * j]), __uint_as_float(draw[2 * j + 1]));
            float lo, hi;
            unpack2(fma2(s2, c2, add2(bias2[pair], nl1)), lo, hi);
            f32x2 p = pack2(ex2(lo), ex2(hi));
            f32x2 dd = add2(d2, nd1);
            if (decltype(drops_keys)::value) {
              p = select2(p, bits, 2 * pair);
              dd = select2(dd, bits, 2 * pair);
            }
            acc2[pair] = fma2(p, dd, acc2[pair]);
          }
        };
        uint32_t s_a[4], d_a[4], s_b[4], d_b[4];
        tmem_ld4(s_t, s_a);
        tmem_ld4(s_t + kTile, d_a);
#pragma unroll
        for (int quad = 0; quad < 8; quad += 2) {
          // the next row's scores are probed half-way through this row: the answer travels under the arithmetic
          if (quad == 4 && i + 1 < n_rows) scores_there = mbar_test(bar(DbSmem::sd_full + (buf ^ 1)), ((i + 1) >> 1) & 1);
          tmem_wait_ld();
          tmem_loaded(s_a);
          tmem_loaded(d_a);
          tmem_ld4(s_t + (quad + 1) * 4, s_b);
          tmem_ld4(s_t + kTile + (quad + 1) * 4, d_b);
          work4(quad, s_a, d_a);
          tmem_wait_ld();
          tmem_loaded(s_b);
          tmem_loaded(d_b);
          if (quad + 2 < 8) {
            tmem_ld4(s_t + (quad + 2) * 4, s_a);
            tmem_ld4(s_t + kTile + (quad + 2) * 4, d_a);
          } else {
            tc_fence_before_sync();
            mbar_arrive_warp(bar(DbSmem::sd_free + buf));
          }
          work4(quad + 1, s_b, d_b);
        }
      };
      if (!BITS || bits == 0xffffffffu)
        row_body(std::false_type{});
      else
        row_body(std::true_type{});
    }
    if (!BITS && key_base + 32 > end) {  // keys that no row keeps
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float lo, hi;
        unpack2(acc2[i], lo, hi);
        acc2[i] = pack2(key_base + 2 * i < end ? lo : 0.f, key_base + 2 * i + 1 < end ? hi : 0.f);
      }
    }
    if (ok && q_valid) {
      if (P.num_parts == 1 && P.dbias_f32) {
        float* dst = reinterpret_cast<float*>(P.dbias) + b * P.db_sb + h * P.db_sh + int64_t(q_index) * P.db_sq +
                     int64_t(key_base) * P.db_sk;
        if (P.db_sk == 1 && key_base + 32 <= P.cols && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float a, b2, c, d;
            unpack2(acc2[2 * i], a, b2);
            unpack2(acc2[2 * i + 1], c, d);
            reinterpret_cast<float4*>(dst)[i] = make_float4(a, b2, c, d);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float lo, hi;
            unpack2(acc2[i], lo, hi);
            if (key_base + 2 * i < P.cols) dst[int64_t(2 * i) * P.db_sk] = lo;
            if (key_base + 2 * i + 1 < P.cols) dst[int64_t(2 * i + 1) * P.db_sk] = hi;
          }
        }
      } else if (P.num_parts == 1) {
        T* dst = reinterpret_cast<T*>(P.dbias) + b * P.db_sb + h * P.db_sh + int64_t(q_index) * P.db_sq + int64_t(key_base) * P.db_sk;
        if (P.db_sk == 1 && key_base + 32 <= P.cols && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            reinterpret_cast<uint4*>(dst)[c] = make_uint4(pack16<T>(acc2[4 * c]), pack16<T>(acc2[4 * c + 1]),
                                                          pack16<T>(acc2[4 * c + 2]), pack16<T>(acc2[4 * c + 3]));
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float lo, hi;
            unpack2(acc2[i], lo, hi);
            if (key_base + 2 * i < P.cols) dst[int64_t(2 * i) * P.db_sk] = T(lo);
            if (key_base + 2 * i + 1 < P.cols) dst[int64_t(2 * i + 1) * P.db_sk] = T(hi);
          }
        }
      } else {
        float* dst = P.parts + (((int64_t(part) * P.batch + b) * P.heads + h) * P.cols + q_index) * P.cols + key_base;
        if (key_base + 32 <= P.cols && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float a, b2, c, d;
            unpack2(acc2[2 * i], a, b2);
            unpack2(acc2[2 * i + 1], c, d);
            reinterpret_cast<float4*>(dst)[i] = make_float4(a, b2, c, d);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float lo, hi;
            unpack2(acc2[i], lo, hi);
            if (key_base + 2 * i < P.cols) dst[2 * i] = lo;
            if (key_base + 2 * i + 1 < P.cols) dst[2 * i + 1] = hi;
          }
        }
      }
    }
  }
}

// No dropped key; keys tested, no list; mask with a list.  Keys behind a ragged end need no test: their sums are not stored.
enum DbRows { kDbAllKept, kDbTested, kDbMasked };

// Rows that keep the same keys of the tile, up to some end, are walked without tests, and without the list where that is all
// rows (tests and list cost 5 to 8 % even where nothing is dropped, tests 20 % and more where they take effect).
template <typename T, int ROWS>
__global__ void __launch_bounds__(kDbThreads, 1) ta_bwd_dbias_kernel(const __grid_constant__ DbParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + DbSmem::abort_flag);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + DbSmem::tmem_slot);
  auto bar = [&](int index) -> uint32_t { return smem_base + DbSmem::bars + index * 8; };

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (device_failed()) return;
  int idx = blockIdx.x;
  const int kt = idx % P.tiles;
  idx /= P.tiles;
  const int qt = idx % P.tiles;
  idx /= P.tiles;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int b = idx % P.batch;
  const int part = idx / P.batch;
  const int row_lo = part * P.rows_per_part;
  const int row_hi = min(P.rows, row_lo + P.rows_per_part);
  const int part_rows = max(0, row_hi - row_lo);
  uint16_t* row_list = reinterpret_cast<uint16_t*>(smem_gen + DbSmem::row_list);
  volatile int* row_count = reinterpret_cast<volatile int*>(smem_gen + DbSmem::row_count);
  // Where the listed rows keep the same keys of the tile, all up to a common end (a mask of real tokens), they are walked
  // without tests and what stands behind the end is not stored; -1 otherwise.
  volatile int* keys_end = reinterpret_cast<volatile int*>(smem_gen + DbSmem::keys_end);
  if (ROWS == kDbMasked && warp == 0) {
    const uint32_t* live = P.live + int64_t(b) * P.rows + row_lo;
    const int64_t all_rows = int64_t(P.batch) * P.rows;
    const uint32_t *full = live + all_rows, *length = live + 2 * all_rows;
    int count = 0;
    bool kept = true;
    uint32_t shortest = ~0u, longest = 0;
#pragma unroll 8
    for (int first = 0; first < part_rows; first += 32) {
      const int i = min(first + lane, part_rows - 1);  // loads without conditions: many in flight
      const uint32_t tiles = __ldg(live + i), whole = __ldg(full + i), keys = __ldg(length + i);
      const bool is_live = first + lane < part_rows && ((tiles >> kt) & 1u) != 0;
      const uint32_t bits = __ballot_sync(0xffffffffu, is_live);
      if (is_live) {
        kept &= ((whole >> kt) & 1u) != 0;
        shortest = min(shortest, keys);
        longest = max(longest, keys);
        row_list[count + __popc(bits & ((1u << lane) - 1))] = uint16_t(i);
      }
      count += __popc(bits);
    }
    kept = __all_sync(0xffffffffu, kept);
    shortest = __reduce_min_sync(0xffffffffu, shortest);
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (lane == 0) {
      *row_count = count;
      *keys_end = kept ? P.cols : shortest == longest && int(longest) >= 0 ? int(longest) : -1;
    }
  }

  if (tid == 0) {
    *abort_flag = 0;
    mbar_init(bar(DbSmem::bias_full), 1);
    for (int i = 0; i < kDbRing; ++i) {
      mbar_init(bar(DbSmem::row_full + i), 1);
      mbar_init(bar(DbSmem::row_empty + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(DbSmem::sd_full + i), 1);
      mbar_init(bar(DbSmem::sd_free + i), kDbElemWarps);
    }
    fence_barrier_init();
  }
  if (warp == kDbMmaWarp) {
    tmem_alloc(smem_base + DbSmem::tmem_slot, 512);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int end = ROWS == kDbMasked ? *keys_end : P.cols;
  const bool kept = end >= 0, whole = kept && (ROWS != kDbMasked || *row_count == part_rows);
  auto walk = [&](auto tests, auto listed) {
    dbias_walk<T, decltype(tests)::value, decltype(listed)::value>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, b, h, qt,
                                                                   kt, part, row_lo, part_rows, kept ? end : P.cols);
  };
  if (ROWS != kDbTested && whole)
    walk(std::false_type{}, std::false_type{});
  else if (ROWS == kDbMasked && kept)
    walk(std::false_type{}, std::true_type{});
  else if (ROWS == kDbMasked)
    walk(std::true_type{}, std::true_type{});
  else if (ROWS == kDbTested)
    walk(std::true_type{}, std::false_type{});
  teardown(abort_flag, tmem_base, kDbMmaWarp, 512);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------

uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }

int64_t padded_cols(const oops_ta_problem& p) { return (int64_t(p.cols) + 7) & ~int64_t(7); }

// Row parts of the shared-bias kernel: one CTA per (part, batch, head, 128 x 128 tile) at one CTA per SM.  The
// smallest part count whose CTAs fill whole waves of the 148 SMs to 90 % is taken (the best one if none does);
// with a single part the kernel stores the final gradient and no partial planes exist.
int bias_parts(const oops_ta_problem& p) {
  const int64_t tiles = ceil_div(p.cols, kTile);
  const int64_t ctas = int64_t(p.batch) * p.heads * tiles * tiles;
  const int limit = (int)std::min<int64_t>(16, p.rows);
  int best = 1;
  double best_fill = 0.0;
  for (int parts = 1; parts <= limit; ++parts) {
    const int64_t total = ctas * parts;
    const double fill = double(total) / double(ceil_div(total, 148) * 148);
    if (fill > best_fill + 1e-9) {
      best = parts;
      best_fill = fill;
    }
    if (fill >= 0.9) return parts;
  }
  return best;
}

// rows of more than 6 query tiles are walked in groups of query tiles by one CTA
int fused_groups(const oops_ta_problem& p) { return (int)ceil_div(ceil_div(p.cols, kTile), kFMaxQTiles); }

// scratch slots that carry the f32 sums of dK and dV from group to group: one per SM id, two tensors, 32 floats per key
int64_t fused_slot_keys(const oops_ta_problem& p) { return ceil_div(p.cols, kTile) * kTile; }
uint64_t fused_slot_bytes(const oops_ta_problem& p) {
  return align256(uint64_t(kFSlots) * 2 * fused_slot_keys(p) * kHeadDim * sizeof(float));
}

// Columns, and items per CTA, from which the single-pass kernel makes the row dots itself.  Its statistics warp takes some 6000 clocks a query tile for them, which
// are hidden under the steps where a row has many: 768 columns 1008 + 50 (prepare_kernel) -> 1032 us, 520 505 + 25 -> 520; 512
// 329 + 24 -> 350, 256 (two samples) 104 + 11 -> 160.  In rows of several groups the first tiles delay a CTA's start (1024: 2842 + 84 -> 3149), and so do
// those of its first item: 768 columns, 1 item a CTA 52 + 2 -> 63, 4 items 198 + 10 -> 215, 6 293 + 16 -> 311, 8 434 + 22 -> 454; 520, 8 306 + 15 -> 320.
constexpr int kOwnDeltaCols = 4 * kTile, kOwnDeltaItems = 8;

// The single-pass kernel serves calls that want dQ together with dK or dV and no per-row bias gradient, on rows
// of up to 4096 columns (32 key tiles, one bit each in the words that describe a row's mask).
bool fused_applies(const oops_ta_problem& p, const oops_ta_grads& g) {
  if ((p.flags & OOPS_TA_FLAG_SPLIT_REVERSE) != 0) return false;
  if (g.dbias && p.bias_groups > 1) return false;
  if (p.cols > kFMaxCols) return false;
  return g.dq.ptr != nullptr && (g.dk.ptr != nullptr || g.dv.ptr != nullptr);
}

// Rows and columns from which the single-pass kernel gets a bias that is closed behind a ragged row's end, or a token mask's.  Ragged: 300 columns 134 -> 124 us, 500
// 347 -> 328, 700 962 -> 912, the copy 3 to 5.  Masks of 94 % of the tokens: 256 columns, two samples 125 -> 113 us and a copy of 3, 200, two samples 91 -> 88 + 3,
// 384 186 -> 170 + 3, 512 375 -> 338 + 4, 1000 3175 -> 2778 + 7; of 80 %: 768 1202 -> 980 + 11, 1400 7855 -> 4849 + 16.  A copy that only tests walk over
// is worth its time in ragged rows, whose own pitch is no multiple of a tile's 128 bytes (scattered keys, 500 columns 399 -> 394 + 4 - 2.5).
constexpr int kClosedCols = 192, kClosedRows = 64;
bool closes_bias(const oops_ta_problem& p, const oops_ta_grads& g) {
  return fused_applies(p, g) && bias_closes(p) && (p.cols % kTile != 0 || (p.mask && p.batch <= kUniformSamples)) && p.cols >= kClosedCols &&
         p.rows >= kClosedRows;
}

// What it takes behind the rest of the scratch: a word per sample, the bias.
uint64_t closing_bytes(const oops_ta_problem& p) { return align256(uint64_t(p.batch) * 4) + closed_bias_bytes(p); }

struct Layout {
  uint64_t delta, live, bias_t, pair_parts, parts, total;
  uint64_t closed;  // behind the rest: `total` does without it
};

Layout workspace_layout(const oops_ta_problem& p, const oops_ta_grads& g) {
  Layout l{};
  uint64_t at = 0;
  l.delta = at;
  at += align256(uint64_t(p.batch) * p.rows * p.heads * p.cols * sizeof(float));
  l.live = at;
  if (p.mask) at += align256(uint64_t(p.batch) * p.rows * sizeof(uint32_t) * 4);
  l.bias_t = at;
  const bool fused = fused_applies(p, g);
  if (p.bias_groups != 0 && (g.dk.ptr || g.dv.ptr) && !fused)
    at += align256(uint64_t(p.batch) * p.bias_groups * p.heads * p.cols * padded_cols(p) * 2);
  l.pair_parts = at;  // per-SM slots of the single-pass kernel (rows of more than one group of query tiles)
  if (fused && fused_groups(p) > 1) at += fused_slot_bytes(p);
  l.parts = at;
  if (g.dbias && p.bias_groups == 1 && bias_parts(p) > 1)
    at += align256(uint64_t(bias_parts(p)) * p.batch * p.heads * p.cols * p.cols * sizeof(float));
  l.total = at;
  l.closed = align256(at);
  return l;
}

template <typename T, typename Params, typename K1, typename K0>
int launch_pair(bool has_bias, K1 with_bias, K0 without_bias, const Params& P, unsigned grid, int smem, cudaStream_t stream,
                const char* what) {
  auto go = [&](auto kernel) -> int {
    const int rc = reserve_smem(kernel, smem);
    if (rc) return rc;
    kernel<<<grid, kThreads, smem, stream>>>(P);
    count_launch();
    return check_launch(what);
  };
  return has_bias ? go(with_bias) : go(without_bias);
}

template <typename T>
int run_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                 const oops_ta_grads& g, cudaStream_t stream) {
  const Layout layout = workspace_layout(p, g);
  if (!p.workspace || p.workspace_bytes < layout.total)
    return fail(OOPS_TA_WORKSPACE_TOO_SMALL, "backward needs %llu scratch bytes, got %llu", (unsigned long long)layout.total,
                (unsigned long long)p.workspace_bytes);
  char* base = reinterpret_cast<char*>(p.workspace);
  float* delta = reinterpret_cast<float*>(base + layout.delta);
  const bool has_bias = p.bias_groups != 0;
  const bool row_bias_grad = g.dbias && p.bias_groups > 1;
  const bool shared_bias_grad = g.dbias && p.bias_groups == 1;
  int status;

  // Key tiles with a kept key, one bit each: rows of more than 32 tiles (which the single-pass kernel does not take) go
  // without, as do calls without a mask.
  uint32_t* live = p.mask && ceil_div(p.cols, kTile) <= 32 ? reinterpret_cast<uint32_t*>(base + layout.live) : nullptr;

  // delta = rowsum(O * dO), unless an earlier call has left it, and what the kernels ask about the mask, which they must find
  // whatever the workspace holds (a second call with a mask: 159 -> 169 us at 96 rows of 768 columns, 1165 -> 1168 at 768).
  const bool fused = fused_applies(p, g);
  const bool words16 = (reinterpret_cast<uintptr_t>(out.ptr) & 15) == 0 && out.sb % 8 == 0 && out.sr % 8 == 0 && out.sc % 8 == 0 && out.sh % 8 == 0;
  const bool own_delta = fused && words16 && (p.flags & OOPS_TA_FLAG_REUSE_DELTA) == 0 && p.cols > kOwnDeltaCols && fused_groups(p) == 1 &&
                         int64_t(p.batch) * p.rows * p.heads >= int64_t(kOwnDeltaItems) * sm_count();
  const int64_t total = (p.flags & OOPS_TA_FLAG_REUSE_DELTA) != 0 || own_delta ? 0 : int64_t(p.batch) * p.rows * p.heads * p.cols;
  const int64_t cells = p.heads > 0 ? total / p.heads : 0;
  const unsigned delta_blocks = (unsigned)ceil_div(cells, 64);
  const unsigned mask_blocks = live ? (unsigned)ceil_div(int64_t(p.batch) * p.rows, 8) : 0u;
  if (delta_blocks + mask_blocks > 0) {
    const int vec_ok = (reinterpret_cast<uintptr_t>(out.ptr) & 15) == 0 && (reinterpret_cast<uintptr_t>(dout.ptr) & 15) == 0 &&
                       out.sb % 8 == 0 && out.sr % 8 == 0 && out.sc % 8 == 0 && out.sh % 8 == 0 && dout.sb % 8 == 0 &&
                       dout.sr % 8 == 0 && dout.sc % 8 == 0 && dout.sh % 8 == 0;
    auto kernel = p.heads == 1 ? prepare_kernel<T, 1> : prepare_kernel<T, 4>;
    kernel<<<delta_blocks + mask_blocks, 256, 0, stream>>>(out, dout, delta, (uint32_t)cells, p.cols, p.heads, p.rows, vec_ok,
                                                           dout.sr < dout.sc, mask_blocks, p.mask, p.mask_sb, p.mask_sr, p.mask_sc, live,
                                                           p.batch * p.rows);
    count_launch();
    status = check_launch("tcgen05 delta");
    if (status) return status;
  }

  if (fused) {
    FParams P{};
    status = encode_pair(&P.map_q, p, p.q, kTile, "query");
    if (!status) status = encode_pair(&P.map_dout, p, dout, kTile, "upstream gradient");
    if (!status) status = encode_pair(&P.map_k, p, p.k, kTile, "key");
    if (!status) status = encode_pair(&P.map_v, p, p.v, kTile, "value");
    P.closed = closes_bias(p, g) && p.workspace_bytes >= layout.closed + closing_bytes(p) && ((reinterpret_cast<uintptr_t>(base) + layout.closed) & 15) == 0;
    if (!status && P.closed) {
      ClosedBiasLook look;
      if (live && p.batch <= kUniformSamples) {
        P.prefix = look.prefix = live + 2 * int64_t(p.batch) * p.rows;
        P.uniform = look.found = reinterpret_cast<uint32_t*>(base + layout.closed);
        look.drops = live + 3 * int64_t(p.batch) * p.rows;
        look.rows = p.rows;
        look.whole = p.cols % kTile == 0;
      }
      P.logits = Logits(p);
      status = close_bias(&P.map_closed, p, base + layout.closed + align256(uint64_t(p.batch) * 4), "bias", stream, look);
    }
    if (!status && has_bias && (!P.closed || p.cols % kTile == 0))  // (over ragged rows every walk takes the closed one)
      status = encode_bias(&P.map_bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
    if (status) return status;
    P.dq = g.dq;
    P.dk = g.dk;
    P.dv = g.dv;
    P.write_dq = g.dq.ptr != nullptr;
    P.write_dk = g.dk.ptr != nullptr;
    P.write_dv = g.dv.ptr != nullptr;
    P.lse = lse;
    P.delta = delta;
    P.out = out;
    P.dout = dout;
    P.own_delta = own_delta;
    P.mask = p.mask;
    P.m_sb = p.mask_sb;
    P.m_sr = p.mask_sr;
    P.m_sc = p.mask_sc;
    P.batch = p.batch;
    P.rows = p.rows;
    P.cols = p.cols;
    P.heads = p.heads;
    P.bias_groups = p.bias_groups;
    P.live = live;
    P.items = p.batch * p.rows * p.heads;
    P.q_tiles = (int)ceil_div(p.cols, kTile);
    P.k_tiles = P.q_tiles;
    P.groups = fused_groups(p);
    P.tiles_per_group = (int)ceil_div(P.q_tiles, P.groups);
    P.scale = p.scale;
    if (P.groups > 1) {
      P.slots = reinterpret_cast<float*>(base + layout.pair_parts);
      P.slot_keys = fused_slot_keys(p);
    }
    // A CTA works through several items where a row is one group of query tiles: the copies and score products of the next
    // item run under the last steps and the read-out of this one (N = 256: 84 -> 68 us).  Rows of several groups keep a CTA
    // to themselves, which sums their dK and dV in its SM's slot.
    const unsigned grid = (unsigned)(P.groups > 1 ? P.items : std::min(P.items, sm_count()));
    auto go = [&](auto kernel) -> int {
      const int rc = reserve_smem(kernel, kFSmemBytes);
      if (rc) return rc;
      kernel<<<grid, kFThreads, kFSmemBytes, stream>>>(P);
      count_launch();
      return check_launch("tcgen05 dQ/dK/dV");
    };
    const bool has_bits = p.mask || (p.cols % kTile != 0 && !P.closed);
    auto pick = [&](auto bias, auto groups) {
      constexpr bool HAS_BIAS = decltype(bias)::value, GROUPS = decltype(groups)::value;
      if constexpr (!GROUPS)
        if (P.q_tiles == 1) return has_bits ? go(ta_bwd_fused_kernel<T, HAS_BIAS, false, true, true>) : go(ta_bwd_fused_kernel<T, HAS_BIAS, false, false, true>);
      return has_bits ? go(ta_bwd_fused_kernel<T, HAS_BIAS, GROUPS, true, false>) : go(ta_bwd_fused_kernel<T, HAS_BIAS, GROUPS, false, false>);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    status = P.groups > 1 ? (has_bias ? pick(Yes{}, Yes{}) : pick(No{}, Yes{})) : (has_bias ? pick(Yes{}, No{}) : pick(No{}, No{}));
    if (status) return status;
  }

  if (!fused && (g.dq.ptr || row_bias_grad)) {
    DqParams P{};
    status = encode_pair(&P.map_q, p, p.q, kTile, "query");
    if (!status) status = encode_pair(&P.map_dout, p, dout, kTile, "upstream gradient");
    if (!status) status = encode_pair(&P.map_k, p, p.k, kStep, "key");
    if (!status) status = encode_pair(&P.map_v, p, p.v, kStep, "value");
    if (!status && has_bias)
      status = encode_bias(&P.map_bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
    if (status) return status;
    P.dq = g.dq;
    P.write_dq = g.dq.ptr != nullptr;
    P.lse = lse;
    P.delta = delta;
    P.mask = p.mask;
    P.m_sb = p.mask_sb;
    P.m_sr = p.mask_sr;
    P.m_sc = p.mask_sc;
    if (row_bias_grad) {
      P.dbias_rows = g.dbias;
      P.db_sb = g.dbias_sb;
      P.db_sg = g.dbias_sg;
      P.db_sh = g.dbias_sh;
      P.db_sq = g.dbias_sq;
      P.db_sk = g.dbias_sk;
    }
    P.batch = p.batch;
    P.rows = p.rows;
    P.cols = p.cols;
    P.heads = p.heads;
    P.bias_groups = p.bias_groups;
    P.q_pairs = (int)ceil_div(p.cols, kTilesPerCta * kTile);
    P.k_steps = (int)ceil_div(p.cols, kStep);
    P.scale = p.scale;
    const unsigned grid = (unsigned)(int64_t(p.batch) * p.rows * p.heads * P.q_pairs);
    status = launch_pair<T>(has_bias, ta_bwd_dq_kernel<T, true>, ta_bwd_dq_kernel<T, false>, P, grid, kDqSmemBytes, stream,
                            "tcgen05 dQ");
    if (status) return status;
  }

  if (!fused && (g.dk.ptr || g.dv.ptr)) {
    DkvParams P{};
    status = encode_pair(&P.map_k, p, p.k, kTile, "key");
    if (!status) status = encode_pair(&P.map_v, p, p.v, kTile, "value");
    if (!status) status = encode_pair(&P.map_q, p, p.q, kStep, "query");
    if (!status) status = encode_pair(&P.map_dout, p, dout, kStep, "upstream gradient");
    if (status) return status;
    if (has_bias) {
      uint16_t* bias_t = reinterpret_cast<uint16_t*>(base + layout.bias_t);
      const int64_t stride = padded_cols(p);
      dim3 grid((unsigned)ceil_div(stride, 32), (unsigned)ceil_div(p.cols, 32), (unsigned)(p.batch * p.bias_groups * p.heads));
      transpose_bias_kernel<<<grid, dim3(32, 8), 0, stream>>>(reinterpret_cast<const uint16_t*>(p.bias), bias_t, p.cols,
                                                              p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, p.heads,
                                                              p.bias_groups, stride);
      count_launch();
      status = check_launch("tcgen05 bias transpose");
      if (status) return status;
      const int64_t plane = int64_t(p.cols) * stride;
      status = encode_bias(&P.map_bias_t, p, bias_t, stride, plane, plane * p.heads, plane * p.heads * p.bias_groups, kTile,
                           "transposed bias");
      if (status) return status;
    }
    P.dk = g.dk;
    P.dv = g.dv;
    P.write_dk = g.dk.ptr != nullptr;
    P.write_dv = g.dv.ptr != nullptr;
    P.lse = lse;
    P.delta = delta;
    P.mask = p.mask;
    P.m_sb = p.mask_sb;
    P.m_sr = p.mask_sr;
    P.m_sc = p.mask_sc;
    P.batch = p.batch;
    P.rows = p.rows;
    P.cols = p.cols;
    P.heads = p.heads;
    P.bias_groups = p.bias_groups;
    P.k_pairs = (int)ceil_div(p.cols, kTilesPerCta * kTile);
    P.q_steps = (int)ceil_div(p.cols, kStep);
    P.scale = p.scale;
    const unsigned grid = (unsigned)(int64_t(p.batch) * p.rows * p.heads * P.k_pairs);
    status = launch_pair<T>(has_bias, ta_bwd_dkv_kernel<T, true>, ta_bwd_dkv_kernel<T, false>, P, grid, kDkvSmemBytes, stream,
                            "tcgen05 dK/dV");
    if (status) return status;
  }

  if (shared_bias_grad) {
    DbParams P{};
    status = encode_pair(&P.map_q, p, p.q, kTile, "query");
    if (!status) status = encode_pair(&P.map_dout, p, dout, kTile, "upstream gradient");
    if (!status) status = encode_pair(&P.map_k, p, p.k, kTile, "key");
    if (!status) status = encode_pair(&P.map_v, p, p.v, kTile, "value");
    if (!status) status = encode_bias(&P.map_bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
    if (status) return status;
    P.num_parts = bias_parts(p);
    P.parts = P.num_parts > 1 ? reinterpret_cast<float*>(base + layout.parts) : nullptr;
    P.dbias = g.dbias;
    P.db_sb = g.dbias_sb;
    P.db_sh = g.dbias_sh;
    P.db_sq = g.dbias_sq;
    P.db_sk = g.dbias_sk;
    P.dbias_f32 = (p.flags & OOPS_TA_FLAG_DBIAS_F32) != 0;
    P.lse = lse;
    P.delta = delta;
    P.mask = p.mask;
    P.m_sb = p.mask_sb;
    P.m_sr = p.mask_sr;
    P.m_sc = p.mask_sc;
    P.batch = p.batch;
    P.rows = p.rows;
    P.cols = p.cols;
    P.heads = p.heads;
    P.tiles = (int)ceil_div(p.cols, kTile);
    P.rows_per_part = (int)ceil_div(p.rows, P.num_parts);
    P.live = live;
    P.scale = p.scale;
    const unsigned grid = (unsigned)(int64_t(P.num_parts) * p.batch * p.heads * P.tiles * P.tiles);
    auto kernel = !p.mask                                   ? ta_bwd_dbias_kernel<T, kDbAllKept>
                  : live && P.rows_per_part <= kDbListRows ? ta_bwd_dbias_kernel<T, kDbMasked>
                                                           : ta_bwd_dbias_kernel<T, kDbTested>;
    status = reserve_smem(kernel, kDbSmemBytes);
    if (status) return status;
    kernel<<<grid, kDbThreads, kDbSmemBytes, stream>>>(P);
    count_launch();
    status = check_launch("tcgen05 shared-bias gradient");
    if (status) return status;
    if (P.num_parts > 1) {
      const int64_t plane = int64_t(p.batch) * p.heads * p.cols * p.cols;
      // (four keys a thread leave a small gradient on a few SMs: 64 columns of four heads, 4.5 us, with one 3.4)
      const int quads = plane >= 512 * int64_t(sm_count()) && p.cols % 4 == 0 && (reinterpret_cast<uintptr_t>(P.parts) & 15) == 0 && g.dbias_sk == 1 &&
                        (reinterpret_cast<uintptr_t>(g.dbias) & 15) == 0 && g.dbias_sb % 4 == 0 &&
                        g.dbias_sh % 4 == 0 && g.dbias_sq % 4 == 0;
      const unsigned blocks = (unsigned)ceil_div(quads ? plane / 4 : plane, 256);
      if (P.dbias_f32)
        reduce_parts_kernel<float><<<blocks, 256, 0, stream>>>(P.parts, P.num_parts, g.dbias, g.dbias_sb, g.dbias_sh, g.dbias_sq, g.dbias_sk,
                                                               p.heads, p.cols, plane, quads);
      else
        reduce_parts_kernel<T><<<blocks, 256, 0, stream>>>(P.parts, P.num_parts, g.dbias, g.dbias_sb, g.dbias_sh, g.dbias_sq, g.dbias_sk,
                                                           p.heads, p.cols, plane, quads);
      count_launch();
      status = check_launch("tcgen05 shared-bias reduce");
      if (status) return status;
    }
  }
  return OOPS_TA_OK;
}

}  // namespace

bool tensor_backward_applies(const oops_ta_problem& p, const oops_ta_grads* g) {
  if (!tensor_forward_applies(p)) return false;
  const int64_t rows = int64_t(p.batch) * p.rows * p.heads * p.cols;
  if (rows > 0x7fffffffll) return false;  // (cell, head) pairs are counted in 32 bits
  (void)g;
  return true;
}

uint64_t tensor_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g) {
  const Layout layout = workspace_layout(p, g);
  return closes_bias(p, g) ? layout.closed + closing_bytes(p) : layout.total;
}

int tensor_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                    const oops_ta_grads& g, cudaStream_t stream) {
  if ((reinterpret_cast<uintptr_t>(dout.ptr) & 15) != 0 || !stride_ok(dout.sb, p.batch) || !stride_ok(dout.sr, p.rows) ||
      !stride_ok(dout.sc, p.cols) || !stride_ok(dout.sh, p.heads))
    return fail(OOPS_TA_UNSUPPORTED_LAYOUT, "upstream gradient must be 16-byte aligned with strides that are multiples of 8");
  if (p.dtype == OOPS_TA_BF16) return run_backward<__nv_bfloat16>(p, out, dout, lse, g, stream);
  return run_backward<__half>(p, out, dout, lse, g, stream);
}

int backward_device_status(int reset) { return read_tu_device_status(reset); }

}  // namespace oops_ta
