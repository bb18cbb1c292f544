// Triangle attention for f32 operands: full-precision FFMA products (the reference's "ieee" mode,
// oops/runtime/dispatch.py:260-328), scores kept on chip.  Definition as in the reference's kernels
// (oops/attention/triangle/triton/kernel.py:128-147 scores, :250-261 normalisation, :499-564 dQ, :682-714 dK/dV).
//
//   forward   CTA = (batch, row, head, 64 queries): 64-key tiles, online softmax, O in registers.
//   reverse   CTA = (batch, row, head): for every 64-key tile (dK, dV in registers) walk the 64-query tiles; S, P, dP
//             and dS are made once and feed all three gradients.  dQ is read, added to and written back by the thread
//             that owns the element (the CTA owns the whole row, so nothing else touches it): five products instead
//             of the seven of separate dQ and dK/dV kernels, fixed order, no atomics.  dS tiles go to scratch when the
//             row-shared bias wants a gradient, and one launch adds them over the rows in a fixed order.
//
// Bound by the FMA pipe, fed from shared memory: 256 threads hold 4 x 4 score elements each and read 8 16-byte words for
// 64 multiply-adds (packed in pairs along the summed axis); rows are 4 floats more than their length apart and a thread's rows
// interleaved, so that no warp-wide read takes more wavefronts than its bytes do.  128 threads with 8 x 4 elements read
// less but held twice the registers: 2 warps per scheduler, which left half of the issue slots empty.  The earlier path wrote the logits of every row to memory
// and read them back for each of seven products.  f32 training call of 64 tokens, 4 heads of 32 channels: 106 us of
// kernels in 12 launches before.
#include <algorithm>

#include "ta_internal.h"

namespace oops_ta {
namespace {

constexpr int kT = 64;             // queries and keys of a tile
constexpr int kThreads = 256;
constexpr int kSPitch = kT + 4;    // floats between the rows of a P or dS tile
constexpr uint64_t kDsBudget = 256ull << 20;  // bytes of dS tiles held for one reduction over rows

struct F32Problem {
  oops_ta_pair q, k, v, out, dout;
  const uint8_t* mask;
  int64_t m_sb, m_sr, m_sc;
  const float* bias;
  int64_t b_sb, b_sg, b_sh, b_sq, b_sk;
  int rows, cols, heads, dim, bias_groups;
  float scale;
  int vec;       // every row of every pair tensor is made of aligned 16-byte words
  int bias_vec;  // so is every row of the bias (its last word may be cut short)
  float* lse;
  oops_ta_pair dq, dk, dv;
  float* delta;
  float* ds;      // [batch][block_rows][heads][cols][cols] (NULL: not wanted)
  float* ds_rows; // per-row bias gradient with its strides (NULL: not wanted)
  int64_t db_sb, db_sg, db_sh, db_sq, db_sk;
  int row0, block_rows;
};

__device__ __forceinline__ float* row_of(const oops_ta_pair& t, int b, int r, int h, int64_t c) {
  return reinterpret_cast<float*>(t.ptr) + b * t.sb + int64_t(r) * t.sr + int64_t(h) * t.sh + c * t.sc;
}

// Asynchronous copies into shared memory; `bytes` of the size are read, the rest is zero.
__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One thread's share of the 64-row tiles of a pair tensor's head: the addresses are worked out once per kernel, a request
// adds the tile's first column.  Rows outside the axis, channels outside the head and columns `keep` drops become zeros.
template <int DP>
struct TileCopy {
  static constexpr int kWords = DP / 4, kRows = kThreads / kWords;  // 16-byte words of a row, rows of one turn
  const float* head;
  int64_t stride;
  int row, c;

  __device__ __forceinline__ TileCopy(const oops_ta_pair& t, int b, int r, int h)
      : head(row_of(t, b, r, h, 0)), stride(t.sc), row(threadIdx.x / kWords), c((threadIdx.x % kWords) * 4) {}

  __device__ __forceinline__ void request(float* dst, const F32Problem& p, int first, const uint8_t* keep) const {
#pragma unroll
    for (int n = 0; n < kT / kRows; ++n) {
      const int col = first + row + n * kRows;
      const bool take = col < p.cols && (!keep || keep[int64_t(col) * p.m_sc] != 0);
      const float* src = head + int64_t(col) * stride + c;
      float* to = dst + (row + n * kRows) * (DP + 4) + c;
      if (p.vec) {
        const bool on = take && c < p.dim;
        copy16(to, on ? src : head, on ? 16 : 0);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool on = take && c + e < p.dim;
          copy4(to + e, on ? src + e : head, on ? 4 : 0);
        }
      }
    }
  }
};

// The same tile with channels as rows of kSPitch floats: dst[c][i].
template <int DP>
struct TransposedCopy {
  static constexpr int kRows = kThreads / DP;
  const float* head;
  int64_t stride;
  int row, c;

  __device__ __forceinline__ TransposedCopy(const oops_ta_pair& t, int b, int r, int h)
      : head(row_of(t, b, r, h, 0)), stride(t.sc), row(threadIdx.x / DP), c(threadIdx.x % DP) {}

  __device__ __forceinline__ void request(float* dst, const F32Problem& p, int first, const uint8_t* keep) const {
    const bool in_head = c < p.dim;
    const float* src = head + int64_t(first + row) * stride + c;
#pragma unroll
    for (int n = 0; n < kT / kRows; ++n, src += kRows * stride) {
      const int col = first + row + n * kRows;
      const bool on = in_head && col < p.cols && (!keep || keep[int64_t(col) * p.m_sc] != 0);
      copy4(dst + c * kSPitch + row + n * kRows, on ? src : head, on ? 4 : 0);
    }
  }
};

// A thread's share of the 64 x 64 tiles of a bias plane (zeros outside).
struct BiasCopy {
  const float* plane;
  int row, c;

  __device__ __forceinline__ BiasCopy(const float* plane_) : plane(plane_), row(threadIdx.x / 16), c((threadIdx.x % 16) * 4) {}

  __device__ __forceinline__ void request(float* dst, const F32Problem& p, int q0, int k0) const {
    if (p.bias_vec) {
      const float* src = plane + int64_t(q0 + row) * p.b_sq + k0 + c;
      const int width = min(4, p.cols - k0 - c) * 4;
#pragma unroll
      for (int n = 0; n < kT / 16; ++n, src += 16 * p.b_sq) {
        const bool on = width > 0 && q0 + row + n * 16 < p.cols;
        copy16(dst + (row + n * 16) * kSPitch + c, on ? src : plane, on ? width : 0);
      }
    } else {
#pragma unroll 4
      for (int i = threadIdx.x; i < kT * kT; i += kThreads) {
        const int q = q0 + i / kT, k = k0 + i % kT;
        const bool on = q < p.cols && k < p.cols;
        copy4(dst + (i / kT) * kSPitch + i % kT, on ? plane + q * p.b_sq + k * p.b_sk : plane, on ? 4 : 0);
      }
    }
  }
};

// s[i][j] = sum_d A[a0 + a_step * i][d] * B[b0 + b_step * j][d] over LEN elements of rows PA and PB floats apart
template <int RI, int RJ, int LEN, int PA, int PB>
__device__ __forceinline__ void dot_rows(const float* A, int a0, int a_step, const float* B, int b0, int b_step, float (&s)[RI][RJ]) {
  float2 acc[RI][RJ];
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < RJ; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int d = 0; d < LEN; d += 4) {
    float4 a[RI], b[RJ];
#pragma unroll
    for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(A + (a0 + a_step * i) * PA + d);
#pragma unroll
    for (int j = 0; j < RJ; ++j) b[j] = *reinterpret_cast<const float4*>(B + (b0 + b_step * j) * PB + d);
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < RJ; ++j) {
        acc[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y), acc[i][j]);
        acc[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w), acc[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < RJ; ++j) s[i][j] = acc[i][j].x + acc[i][j].y;
}

// acc[i][0 .. 3] += sum_k P[row0 + step * i][k] * B[k][c .. c + 3] over the 64 keys of a tile
template <int DP, int R>
__device__ __forceinline__ void rows_times_tile(const float* P, const float* B, int row0, int step, int c, float (&acc)[R][4]) {
#pragma unroll 2
  for (int k = 0; k < kT; k += 4) {
    float4 b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = *reinterpret_cast<const float4*>(B + (k + e) * (DP + 4) + c);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(P + (row0 + step * i) * kSPitch + k);
      const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[i][0] = fmaf(av[e], b[e].x, acc[i][0]);
        acc[i][1] = fmaf(av[e], b[e].y, acc[i][1]);
        acc[i][2] = fmaf(av[e], b[e].z, acc[i][2]);
        acc[i][3] = fmaf(av[e], b[e].w, acc[i][3]);
      }
    }
  }
}

// acc[i][0 .. 3] += sum_q P[q][row0 + i] * B[q][c .. c + 3]: the transposed product, a thread's R columns contiguous
template <int DP, int R>
__device__ __forceinline__ void columns_times_tile(const float* P, const float* B, int row0, int c, float (&acc)[R][4]) {
#pragma unroll 4
  for (int q = 0; q < kT; ++q) {
    const float4 b = *reinterpret_cast<const float4*>(B + q * (DP + 4) + c);
    float a[R];
    if constexpr (R == 2) {
      const float2 v = *reinterpret_cast<const float2*>(P + q * kSPitch + row0);
      a[0] = v.x; a[1] = v.y;
    } else {
#pragma unroll
      for (int i = 0; i < R; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(P + q * kSPitch + row0 + i);
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      acc[i][0] = fmaf(a[i], b.x, acc[i][0]);
      acc[i][1] = fmaf(a[i], b.y, acc[i][1]);
      acc[i][2] = fmaf(a[i], b.z, acc[i][2]);
      acc[i][3] = fmaf(a[i], b.w, acc[i][3]);
    }
  }
}

__device__ __forceinline__ void store4(float* dst, int c, const F32Problem& p, const float (&v)[4], float f) {
  if (p.vec) {
    if (c < p.dim) *reinterpret_cast<float4*>(dst + c) = make_float4(v[0] * f, v[1] * f, v[2] * f, v[3] * f);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < p.dim) dst[c + e] = v[e] * f;
  }
}

__device__ __forceinline__ const float* bias_plane(const F32Problem& p, int b, int r, int h) {
  return p.bias ? p.bias + b * p.b_sb + int64_t(p.bias_groups == 1 ? 0 : r) * p.b_sg + h * p.b_sh : nullptr;
}

template <int DP>
constexpr int tile_floats() { return kT * (DP + 4); }

template <int DP>
__global__ void __launch_bounds__(kThreads) f32_forward_kernel(const F32Problem p) {
  extern __shared__ __align__(16) float f32_smem[];
  float* Q = f32_smem;
  float* K = Q + tile_floats<DP>();
  float* V = K + tile_floats<DP>();
  float* P = V + DP * kSPitch;  // V is held with channels as rows
  float* factor = P + kT * kSPitch;  // [64] rescale factor of a query row
  constexpr int R = DP / 16, kCols = DP / 4;  // O: R rows of four channels per thread, kCols apart; kCols threads per row
  int idx = blockIdx.x;
  const int tiles = (p.cols + kT - 1) / kT, qt = idx % tiles;
  idx /= tiles;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int r = idx % p.rows, b = idx / p.rows;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, oc = tid % kCols, oq = tid / kCols;
  const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;

  const float* plane = bias_plane(p, b, r, h);
  float m[4], l[4], o[R][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
#pragma unroll
  for (int i = 0; i < R; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  // Single buffers: K of the next tile is requested once the scores are made, V and the bias (whose tile the
  // probabilities overwrite in place) once the products with V are, so every copy runs under the other half of the step.
  const TileCopy<DP> k_copy(p.k, b, r, h);
  const TransposedCopy<DP> v_copy(p.v, b, r, h);
  const BiasCopy bias_copy(plane);
  TileCopy<DP>(p.q, b, r, h).request(Q, p, qt * kT, nullptr);
  k_copy.request(K, p, 0, keep);
  copies_commit();
  v_copy.request(V, p, 0, keep);
  if (plane) bias_copy.request(P, p, qt * kT, 0);
  copies_commit();

  for (int kt = 0; kt < tiles; ++kt) {
    const int k0 = kt * kT;
    bool kept[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = k0 + tx + 16 * j;
      kept[j] = key < p.cols && (!keep || keep[int64_t(key) * p.m_sc] != 0);
    }
    copies_wait<1>();
    __syncthreads();
    float s[4][4];
    dot_rows<4, 4, DP, DP + 4, DP + 4>(Q, ty, 16, K, tx, 16, s);
    copies_wait<0>();
    __syncthreads();
    if (kt + 1 < tiles) k_copy.request(K, p, k0 + kT, keep);
    copies_commit();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* row = P + (ty + 16 * i) * kSPitch + tx;
      float peak = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= p.scale;
        if (plane) s[i][j] += row[16 * j];
        if (!kept[j]) s[i][j] = -INFINITY;
        peak = fmaxf(peak, s[i][j]);
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, x));
      const float before = m[i];
      m[i] = fmaxf(before, peak);
      const float base = m[i] == -INFINITY ? 0.f : m[i], shrink = expf(before - base);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = expf(s[i][j] - base);
        row[16 * j] = e;
        sum += e;
      }
      l[i] = l[i] * shrink + sum;
      if (tx == 0) factor[ty + 16 * i] = shrink;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float f = factor[oq + kThreads / kCols * i];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] *= f;
    }
    float add[R][4];
    dot_rows<R, 4, kT, kSPitch, kSPitch>(P, oq, kThreads / kCols, V, oc, kCols, add);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] += add[i][e];
    __syncthreads();
    if (kt + 1 < tiles) {
      v_copy.request(V, p, k0 + kT, keep);
      if (plane) bias_copy.request(P, p, qt * kT, k0 + kT);
    }
    copies_commit();
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
    if (tx == 0) {
      factor[ty + 16 * i] = l[i] > 0.f || l[i] != l[i] ? 1.f / l[i] : 0.f;
      const int q = qt * kT + ty + 16 * i;
      if (p.lse && q < p.cols)
        p.lse[((int64_t(b) * p.rows + r) * p.heads + h) * p.cols + q] = l[i] > 0.f || l[i] != l[i] ? m[i] + logf(l[i]) : 0.f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = oq + kThreads / kCols * i, q = qt * kT + row;
    if (q >= p.cols) continue;
    float* dst = row_of(p.out, b, r, h, q);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (oc + kCols * e < p.dim) dst[oc + kCols * e] = o[i][e] * factor[row];
  }
}

template <int DP>
__global__ void __launch_bounds__(kThreads, 2) f32_backward_kernel(const F32Problem p) {
  extern __shared__ __align__(16) float f32_smem[];
  float* rows2 = f32_smem;  // [2] Q and dO of a query tile
  float* K = rows2 + 4 * tile_floats<DP>();
  float* V = K + tile_floats<DP>();
  float* P = V + tile_floats<DP>();
  float* dS = P + kT * kSPitch;
  float* stats = dS + kT * kSPitch;  // [2][64] lse and delta of the query tile
    // dK and dV: half of the threads each, R rows of four channels; dQ: all threads, RQ rows kStep apart
  constexpr int R = DP / 8, RQ = DP / 16, kCols = DP / 4, kStep = kThreads / kCols;
  int idx = blockIdx.x;
  const int tiles = (p.cols + kT - 1) / kT;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int rr = idx % p.block_rows, b = idx / p.block_rows, r = p.row0 + rr;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, oc = (tid % kCols) * 4, orow = (tid & 127) / kCols, qrow = tid / kCols;
  const bool makes_dv = tid < kThreads / 2;
  const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;
  const int64_t stat_at = ((int64_t(b) * p.rows + r) * p.heads + h) * p.cols;
  float* ds_plane = p.ds ? p.ds + (int64_t(b) * p.block_rows + rr) * p.heads * p.cols * p.cols + int64_t(h) * p.cols * p.cols : nullptr;
  float* ds_row = p.ds_rows ? p.ds_rows + b * p.db_sb + int64_t(r) * p.db_sg + h * p.db_sh : nullptr;

  const float* plane = bias_plane(p, b, r, h);
  const TileCopy<DP> q_copy(p.q, b, r, h), do_copy(p.dout, b, r, h);
  const BiasCopy bias_copy(plane);
  auto request_rows = [&](int step, int qt) {
    float* at = rows2 + (step & 1) * 2 * tile_floats<DP>();
    q_copy.request(at, p, qt * kT, nullptr);
    do_copy.request(at + tile_floats<DP>(), p, qt * kT, nullptr);
  };
  request_rows(0, 0);
  int step = 0;

  for (int kt = 0; kt < tiles; ++kt) {
    const int k0 = kt * kT;
    TileCopy<DP>(p.k, b, r, h).request(K, p, k0, keep);
    TileCopy<DP>(p.v, b, r, h).request(V, p, k0, keep);
    bool kept[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = k0 + tx + 16 * j;
      kept[j] = key < p.cols && (!keep || keep[int64_t(key) * p.m_sc] != 0);
    }
    float acc[R][4];  // dV or dK of the key tile
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;

    for (int qt = 0; qt < tiles; ++qt, ++step) {
      const int q0 = qt * kT;
      const float* Q = rows2 + (step & 1) * 2 * tile_floats<DP>();
      const float* dO = Q + tile_floats<DP>();
      // (the rows of this step, and K and V of a new key tile, were requested before the last barrier)
      if (kt == 0) TileCopy<DP>(p.out, b, r, h).request(P, p, q0, nullptr);  // P is free until the scores of this step
      copies_commit();
      if (plane) bias_copy.request(dS, p, q0, k0);  // dS overwrites the bias in place
      copies_commit();
      float lse = INFINITY, delta = 0.f;
      if (tid < kT && q0 + tid < p.cols) {
        lse = p.lse[stat_at + q0 + tid];
        if (kt > 0) delta = p.delta[stat_at + q0 + tid];  // written by this thread for the first key tile
      }
      copies_wait<1>();
      __syncthreads();
      if (tid < kT) {
        if (kt == 0) {
          for (int d = 0; d < DP; d += 4) {
            const float4 a = *reinterpret_cast<const float4*>(P + tid * (DP + 4) + d);
            const float4 g = *reinterpret_cast<const float4*>(dO + tid * (DP + 4) + d);
            delta += a.x * g.x + a.y * g.y + a.z * g.z + a.w * g.w;
          }
          if (q0 + tid < p.cols) p.delta[stat_at + q0 + tid] = delta;
        }
        stats[tid] = lse;
        stats[kT + tid] = delta;
      }
      float s[4][4];
      dot_rows<4, 4, DP, DP + 4, DP + 4>(Q, ty, 16, K, tx, 16, s);
      copies_wait<0>();
      __syncthreads();
      {  // the next step's rows travel under the rest of this one
        const bool last = qt + 1 == tiles;
        if (!last || kt + 1 < tiles) request_rows(step + 1, last ? 0 : qt + 1);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float norm = stats[ty + 16 * i];
        const int at = (ty + 16 * i) * kSPitch + tx;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x = s[i][j] * p.scale;
          if (plane) x += dS[at + 16 * j];
          s[i][j] = kept[j] ? expf(x - norm) : 0.f;
          P[at + 16 * j] = s[i][j];
        }
      }
      {
        float dp[4][4];
        dot_rows<4, 4, DP, DP + 4, DP + 4>(dO, ty, 16, V, tx, 16, dp);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float shift = stats[kT + ty + 16 * i];
          const int q = q0 + ty + 16 * i;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float ds = kept[j] ? s[i][j] * (dp[i][j] - shift) : 0.f;
            dS[(ty + 16 * i) * kSPitch + tx + 16 * j] = ds;
            const int key = k0 + tx + 16 * j;
            if (q < p.cols && key < p.cols) {
              if (ds_plane) ds_plane[int64_t(q) * p.cols + key] = ds;
              if (ds_row) ds_row[int64_t(q) * p.db_sq + int64_t(key) * p.db_sk] = ds;
            }
          }
        }
      }
      __syncthreads();
      if (p.dq.ptr) {
        // sums of the earlier key tiles, unscaled until the last one; requested ahead of the product they are added to
        float dq[RQ][4], before[RQ][4];
#pragma unroll
        for (int i = 0; i < RQ; ++i) {
          const int q = q0 + qrow + kStep * i;
          const float* src = row_of(p.dq, b, r, h, q);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            dq[i][e] = before[i][e] = 0.f;
            if (kt > 0 && q < p.cols && oc + e < p.dim) before[i][e] = src[oc + e];
          }
        }
        rows_times_tile<DP, RQ>(dS, K, qrow, kStep, oc, dq);
        const float f = kt + 1 == tiles ? p.scale : 1.f;
#pragma unroll
        for (int i = 0; i < RQ; ++i) {
          const int q = q0 + qrow + kStep * i;
#pragma unroll
          for (int e = 0; e < 4; ++e) dq[i][e] += before[i][e];
          if (q < p.cols) store4(row_of(p.dq, b, r, h, q), oc, p, dq[i], f);
        }
      }
      if (makes_dv ? p.dv.ptr != nullptr : p.dk.ptr != nullptr)
        columns_times_tile<DP, R>(makes_dv ? P : dS, makes_dv ? dO : Q, orow * R, oc, acc);
      __syncthreads();  // P, dS, these rows and, after the last query tile, K and V may be overwritten
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int key = k0 + orow * R + i;
      if (key >= p.cols) continue;
      // a dropped key gets exact zeros, whatever its rows and the upstream gradient hold
      const bool dropped = keep && keep[int64_t(key) * p.m_sc] == 0;
      if (dropped) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
      }
      const oops_ta_pair& to = makes_dv ? p.dv : p.dk;
      if (to.ptr) store4(row_of(to, b, r, h, key), oc, p, acc[i], makes_dv ? 1.f : p.scale);
    }
  }
}

// dbias[b][h][q][k] (+)= sum over the block's rows of dS: a CTA takes 32 neighbouring elements, its eight warps every
// eighth row each, and the eight sums are added in warp order.
__global__ void __launch_bounds__(256) f32_bias_sum_kernel(const float* __restrict__ ds, float* __restrict__ dbias, int64_t sb,
                                                           int64_t sh, int64_t sq, int64_t sk, int heads, int cols, int block_rows,
                                                           int64_t total, int add) {
  __shared__ float sums[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = int64_t(blockIdx.x) * 32 + lane, plane = int64_t(cols) * cols;
  const int64_t e = i % plane, bh = i / plane;
  const int h = int(bh % heads);
  const int64_t b = bh / heads;
  float sum = 0.f;
  if (i < total) {
    const float* at = ds + (b * block_rows * heads + h) * plane + e;
#pragma unroll 4
    for (int rr = warp; rr < block_rows; rr += 8) sum += at[int64_t(rr) * heads * plane];
  }
  sums[warp][lane] = sum;
  __syncthreads();
  if (warp == 0 && i < total) {
#pragma unroll
    for (int w = 1; w < 8; ++w) sum += sums[w][lane];
    float* dst = dbias + b * sb + h * sh + (e / cols) * sq + (e % cols) * sk;
    *dst = add ? *dst + sum : sum;
  }
}

bool words_ok(const oops_ta_pair& t) {
  return !t.ptr || ((reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 4 == 0 && t.sr % 4 == 0 && t.sc % 4 == 0 && t.sh % 4 == 0);
}

F32Problem describe(const oops_ta_problem& p) {
  F32Problem f{};
  f.q = p.q;
  f.k = p.k;
  f.v = p.v;
  f.mask = p.mask;
  f.m_sb = p.mask_sb;
  f.m_sr = p.mask_sr;
  f.m_sc = p.mask_sc;
  if (p.bias_groups) {
    f.bias = reinterpret_cast<const float*>(p.bias);
    f.b_sb = p.bias_sb;
    f.b_sg = p.bias_sg;
    f.b_sh = p.bias_sh;
    f.b_sq = p.bias_sq;
    f.b_sk = p.bias_sk;
    f.bias_vec = p.bias_sk == 1 && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0 && p.bias_sb % 4 == 0 && p.bias_sg % 4 == 0 &&
                 p.bias_sh % 4 == 0 && p.bias_sq % 4 == 0;
  }
  f.rows = p.rows;
  f.cols = p.cols;
  f.heads = p.heads;
  f.dim = p.head_dim;
  f.bias_groups = p.bias_groups;
  f.scale = p.scale;
  return f;
}

template <typename Kernel>
int launch(Kernel kernel, const F32Problem& f, int64_t grid, int floats, cudaStream_t stream, const char* what) {
  const int smem = floats * int(sizeof(float));
  const int status = reserve_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (status) return status;
  kernel<<<(unsigned)grid, kThreads, smem, stream>>>(f);
  count_launch();
  return check_launch(what);
}

template <typename F>
int by_width(int dim, F&& run) {
  if (dim <= 16) return run(std::integral_constant<int, 16>{});
  if (dim <= 32) return run(std::integral_constant<int, 32>{});
  return run(std::integral_constant<int, 64>{});
}

uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }

int ds_block_rows(const oops_ta_problem& p) {
  const uint64_t per_row = uint64_t(p.batch) * p.heads * p.cols * p.cols * sizeof(float);
  return (int)std::min<uint64_t>(std::max<uint64_t>(1, kDsBudget / per_row), (uint64_t)p.rows);
}

bool wants_ds(const oops_ta_problem& p, const oops_ta_grads& g) { return g.dbias && p.bias_groups == 1; }

}  // namespace

// Head sizes above 64 would not leave room for two CTAs per SM: they stay with the kernels that keep logits in memory.
bool f32_forward_applies(const oops_ta_problem& p) {
  return p.dtype == OOPS_TA_F32 && p.head_dim <= 64 &&
         int64_t(p.batch) * p.rows * p.heads * ceil_div(p.cols, kT) <= 0x7fffffffll;
}

// A CTA of the reverse pass owns a whole row of a head, so a launch must have enough of those; rows that the dS budget splits
// over launches count by the launch, and pay for every launch's tail.  Against the kernels that split every row into tiles,
// reverse call with 4 heads and a shared-bias gradient (16 / 32 / 64 channels): 112 CTAs a launch (768 columns) take 0.65 /
// 0.78 / 0.89 of their time, 80 (896) 0.85 / 1.03 / 1.18, 48 (1152) 1.36 / 1.66 / 1.91, 16 (2048) 2.6 / 3.2 / 3.9.  In one launch
// 76 take 0.78 (512 columns), 74 0.75 (1024 columns, no bias gradient).
bool f32_backward_applies(const oops_ta_problem& p, const oops_ta_grads& g) {
  if (!f32_forward_applies(p)) return false;
  const int rows = wants_ds(p, g) ? ds_block_rows(p) : p.rows;
  return int64_t(p.batch) * rows * p.heads >= (rows < p.rows ? 96 : 74);
}

uint64_t f32_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g) {
  uint64_t total = align256(uint64_t(p.batch) * p.rows * p.heads * p.cols * sizeof(float));
  if (wants_ds(p, g)) total += align256(uint64_t(p.batch) * ds_block_rows(p) * p.heads * p.cols * p.cols * sizeof(float));
  return total;
}

int f32_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream) {
  F32Problem f = describe(p);
  f.out = out;
  f.lse = lse;
  f.vec = p.head_dim % 4 == 0 && words_ok(p.q) && words_ok(p.k) && words_ok(p.v) && words_ok(out);
  const int64_t grid = int64_t(p.batch) * p.rows * p.heads * ceil_div(p.cols, kT);
  return by_width(p.head_dim, [&](auto width) {
    constexpr int DP = decltype(width)::value;
    return launch(f32_forward_kernel<DP>, f, grid, 2 * tile_floats<DP>() + (DP + kT) * kSPitch + kT, stream, "f32 forward");
  });
}

int f32_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                 const oops_ta_grads& g, cudaStream_t stream) {
  const uint64_t need = f32_backward_workspace(p, g);
  if (p.workspace_bytes < need || !p.workspace)
    return fail(OOPS_TA_WORKSPACE_TOO_SMALL, "backward needs %llu scratch bytes, got %llu", (unsigned long long)need,
                (unsigned long long)p.workspace_bytes);
  F32Problem f = describe(p);
  f.out = out;
  f.dout = dout;
  f.lse = const_cast<float*>(lse);
  f.dq = g.dq;
  f.dk = g.dk;
  f.dv = g.dv;
  f.vec = p.head_dim % 4 == 0;
  for (const oops_ta_pair* t : {&p.q, &p.k, &p.v, &out, &dout, &g.dq, &g.dk, &g.dv}) f.vec = f.vec && words_ok(*t);
  f.delta = reinterpret_cast<float*>(p.workspace);
  const bool summed = wants_ds(p, g);
  if (summed)
    f.ds = reinterpret_cast<float*>(reinterpret_cast<char*>(p.workspace) + align256(uint64_t(p.batch) * p.rows * p.heads * p.cols * sizeof(float)));
  if (g.dbias && !summed) {
    f.ds_rows = reinterpret_cast<float*>(g.dbias);
    f.db_sb = g.dbias_sb;
    f.db_sg = g.dbias_sg;
    f.db_sh = g.dbias_sh;
    f.db_sq = g.dbias_sq;
    f.db_sk = g.dbias_sk;
  }
  const int block = summed ? ds_block_rows(p) : p.rows;
  for (int row0 = 0; row0 < p.rows; row0 += block) {
    f.row0 = row0;
    f.block_rows = std::min(block, p.rows - row0);
    int status = by_width(p.head_dim, [&](auto width) {
      constexpr int DP = decltype(width)::value;
      return launch(f32_backward_kernel<DP>, f, int64_t(p.batch) * f.block_rows * p.heads,
                    6 * tile_floats<DP>() + 2 * kT * kSPitch + 2 * kT, stream, "f32 backward");
    });
    if (status) return status;
    if (summed) {
      const int64_t total = int64_t(p.batch) * p.heads * p.cols * p.cols;
      f32_bias_sum_kernel<<<(unsigned)ceil_div(total, 32), 256, 0, stream>>>(
          f.ds, reinterpret_cast<float*>(g.dbias), g.dbias_sb, g.dbias_sh, g.dbias_sq, g.dbias_sk, p.heads, p.cols, f.block_rows, total,
          row0 > 0);
      count_launch();
      status = check_launch("f32 shared-bias sum");
      if (status) return status;
    }
  }
  return OOPS_TA_OK;
}

}  // namespace oops_ta
