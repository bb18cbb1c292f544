// tcgen05 / TMEM / TMA attention kernels for bf16 operands with head sizes up to 64 other than 32 (multiples of 8): token
// attention with a pair bias.  Definition as in the reference's kernels (oops/attention/triangle/triton/kernel.py:128-147,
// :250-261, :499-564, :682-714, :856).
//
// Probabilities and dS enter their products as a pair of bf16 numbers, value and remainder (16 digits), as in the register-level
// kernels beside this file, which serve f16 (whose exponents need a running scale per row), masks, f32 biases and unaligned
// layouts.  Both numbers go to tensor memory, into the very columns that held the f32 scores they were made from: of
// sixteen columns of scores the first eight become values, the other eight remainders, so that a K = 16 step of the product
// reads its A operand eight columns apart and nothing passes through shared memory.
//
//   forward   CTA = (batch, row, head, 128 queries): a warpgroup whose threads own a query each, a producer warp, an issuing warp;
//             64-key steps, scores in two buffers.
//   reverse   one launch, three kinds of CTA, 64-column steps, two CTAs per SM: dK and dV of 128 keys (scores transposed, a thread
//             owns a key), dQ of 128 queries, and a 128 x 64 tile of the row-shared bias gradient with the rows innermost,
//             summed in registers.  Each makes the scores it needs again, as token attention has too few rows and heads to
//             give a CTA a whole row; nothing is added across CTAs, so results are reproducible.
// What bounds them is the chain of a step (scores, element-wise work, sums, and the trips between them), which the second CTA of an
// SM runs under; no unit is full (counters of 4 samples, 16 heads of 64 channels and 512 tokens: tensor pipe 15 % busy forward and 20 % in the
// reverse, issue slots 28 and 35 %, special-function units 21 and 22 %).  That call took 35 us forward and 136 reverse at register
// level, and takes 14 and 57 here, with the same errors against f64 (1.66e-3 of every result's norm, its rounding).  With queries as rows the next
// scores are issued ahead of the sums (dP has a second buffer there): 24 -> 22 us for dQ alone.  Masks are not served: a step has no place yet for the
// test of a mask tile.
#include <algorithm>
#include <type_traits>

#include "ta_tensor_common.cuh"

namespace oops_ta {
namespace {

using namespace ptx;
using Half = Half2<__nv_bfloat16>;

constexpr int kDim = 64;                        // channels of a tile; channels above the head size are zeros
constexpr int kStep = 64;                       // columns of a step
constexpr int kRowTile = kTile * kDim * 2;      // 128 rows
constexpr int kColTile = kStep * kDim * 2;      // 64 columns
constexpr int kBiasTile = kTile * kStep * 2;
constexpr int kTmemCols = 256;                  // two CTAs share an SM

struct WideParams {
  CUtensorMap row0, row1;    // boxes of 128 rows of the pair tensors: Q, dO (forward: Q)
  CUtensorMap key0, key1;    // boxes of 128 rows: K, V
  CUtensorMap col_q, col_d;  // boxes of 64 rows: Q, dO
  CUtensorMap col_k, col_v;  // boxes of 64 rows: K, V
  CUtensorMap bias;          // box of 128 queries x 64 keys
  CUtensorMap bias_t;        // box of 64 queries x 128 keys, not swizzled
  oops_ta_pair out, dq, dk, dv;
  const void* bias_ptr;
  int64_t b_sb, b_sh, b_sq;
  void* dbias;
  float* parts;
  int64_t db_sb, db_sh, db_sq, db_sk;
  float* lse;
  const float* delta;
  int batch, rows, cols, heads, dim, bias_groups;
  int row_tiles, steps;        // 128-row tiles and 64-column steps of the axis
  int num_parts, rows_per_part, dbias_f32, store_words;
  int dkv_ctas, dq_ctas;
  float scale;
};

// K-major operand (channels contiguous, 128-byte rows): 8-row groups 1024 bytes apart, 32 bytes per 16-channel step.
__device__ __forceinline__ uint64_t k_major(uint32_t at) { return smem_desc(at, 16, 1024, kSwizzle128B); }
constexpr uint64_t kChannelStep = 32 >> 4;
// The same tile as B operand of a product over its rows (MN-major): 16 rows are 2048 bytes.
constexpr uint64_t kRowStep = 2048 >> 4;

// D (128 x 64) = A (128 rows) B (64 rows)^T over the channels; `steps` of 16 channels.
__device__ __forceinline__ void score_product(uint32_t d, uint64_t a, uint64_t b, int steps) {
  constexpr uint32_t idesc = instr_desc(Half::kFormat, 0, 0, kTile, kStep);
  for (int kk = 0; kk < steps; ++kk) mma_ss(d, a + kk * kChannelStep, b + kk * kChannelStep, idesc, kk > 0 ? 1u : 0u);
}
// acc (128 x channels) += W (128 x 64, values and remainders in tensor memory) X (64 rows x channels)
__device__ __forceinline__ void sum_product(uint32_t acc, uint32_t w, uint64_t x, bool first) {
  constexpr uint32_t idesc = instr_desc(Half::kFormat, 0, 1, kTile, kDim);
#pragma unroll
  for (int kk = 0; kk < kStep / 16; ++kk) {
    mma_ts(acc, w + kk * 16, x + kk * kRowStep, idesc, first && kk == 0 ? 0u : 1u);
    mma_ts(acc, w + kk * 16 + 8, x + kk * kRowStep, idesc, 1u);
  }
}

// Sixteen values of a row as eight words of values and eight of remainders.
__device__ __forceinline__ void split16(const f32x2 (&w)[8], uint32_t (&words)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    words[i] = Half::pack(w[i].x, w[i].y);
    const f32x2 rest = fma2(Half::widen(words[i]), pack2(-1.f, -1.f), w[i]);
    words[8 + i] = Half::pack(rest.x, rest.y);
  }
}

// exp(score * scale + bias + norm), norm = -lse: the logit is made as the forward pass makes it, and the norm comes off before the
// change of base, so that a row whose logits are all far from zero sees them cancel.
__device__ __forceinline__ f32x2 probability(f32x2 score, f32x2 scale, f32x2 bias, f32x2 norm) {
  const f32x2 x = mul2(add2(fma2(score, scale, bias), norm), pack2(kLog2e, kLog2e));
  return pack2(ex2(x.x), ex2(x.y));
}

// Channels first .. first + 31 of a row of the result.
__device__ __forceinline__ void store_channels(const oops_ta_pair& to, int dim, int b, int r, int h, int at, int first, const uint32_t (&acc)[32],
                                               float scale) {
  __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(to.ptr) + b * to.sb + int64_t(r) * to.sr + int64_t(h) * to.sh + int64_t(at) * to.sc + first;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (first + 8 * c >= dim) break;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = Half::pack(__uint_as_float(acc[8 * c + 2 * i]) * scale, __uint_as_float(acc[8 * c + 2 * i + 1]) * scale);
    reinterpret_cast<uint4*>(row)[c] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
struct WideFwdSmem {
  static constexpr int q = 0;
  static constexpr int k = q + kRowTile;          // [3]
  static constexpr int v = k + 3 * kColTile;      // [2]
  static constexpr int bias = v + 2 * kColTile;   // [2]
  static constexpr int bars = bias + 2 * kBiasTile;
  static constexpr int q_full = 0;
  static constexpr int k_full = 1, k_empty = 4;   // [3]
  static constexpr int v_full = 7, v_empty = 9;   // [2] with the bias tile of the step
  static constexpr int s_full = 11;               // [2] scores are in tensor memory
  static constexpr int p_full = 13;               // [2] probabilities have taken their place
  // [2] the value product of the step has completed (a barrier per buffer: waiters may be two steps behind the last product, and a
  // parity tells a phase from its neighbours only)
  static constexpr int pv_done = 15;
  static constexpr int num_bars = 17;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int failed = abort_flag + 4;   // a kernel before this one has given up a wait
  static constexpr int bytes = failed + 4 + 1024;
};
constexpr int kWideFwdThreads = 192;
static_assert(WideFwdSmem::bytes <= 113 * 1024, "two forward CTAs must fit in one SM's shared memory");

template <bool HAS_BIAS>
__global__ void __launch_bounds__(kWideFwdThreads, 2) ta_wide_fwd_kernel(const __grid_constant__ WideParams P) {
  using Smem = WideFwdSmem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Smem::abort_flag);
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int idx = int(blockIdx.x);
  const int q0 = idx % P.row_tiles * kTile;
  idx /= P.row_tiles;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int r = idx % P.rows, b = idx / P.rows;
  if (warp == 4) {
    const bool failed = device_failed();  // (looked at beside the other preparations)
    if (lane < Smem::num_bars) {
      int arrivals = 1;
      if (lane >= Smem::v_empty && lane < Smem::s_full) arrivals = HAS_BIAS ? 5 : 1;  // the value product, and the warps' look at the bias
      if (lane >= Smem::p_full && lane < Smem::pv_done) arrivals = 4;
      mbar_init(bar(lane), arrivals);
    }
    fence_barrier_init();
    if (lane == 0) {
      *abort_flag = 0;
      *reinterpret_cast<volatile int*>(smem_gen + Smem::failed) = failed ? 1 : 0;
    }
  }
  if (warp == 5) {
    tmem_alloc(smem_base + Smem::tmem_slot, kTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_gen + Smem::tmem_slot);
  constexpr int kOCol = 2 * kStep;  // scores [2] x 64 | output 64
  const int steps = P.steps;

  if (*reinterpret_cast<volatile int*>(smem_gen + Smem::failed) != 0) {
    // nothing has been requested: on to the end
  } else if (warp == 4) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(bar(Smem::q_full), kRowTile);
      tma_load_5d(smem_base + Smem::q, &P.row0, bar(Smem::q_full), 0, h, q0, r, b);
      for (int i = 0; i < steps && ok; ++i) {
        const int ks = i % 3, vs = i & 1;
        if (i >= 3) ok = mbar_wait(bar(Smem::k_empty + ks), (i / 3 - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(Smem::k_full + ks), kColTile);
        tma_load_5d(smem_base + Smem::k + ks * kColTile, &P.col_k, bar(Smem::k_full + ks), 0, h, i * kStep, r, b);
        if (i >= 2) ok = mbar_wait(bar(Smem::v_empty + vs), (i / 2 - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(Smem::v_full + vs), kColTile + (HAS_BIAS ? kBiasTile : 0));
        if (HAS_BIAS)
          tma_load_5d(smem_base + Smem::bias + vs * kBiasTile, &P.bias, bar(Smem::v_full + vs), i * kStep, q0, h, P.bias_groups == 1 ? 0 : r, b);
        tma_load_5d(smem_base + Smem::v + vs * kColTile, &P.col_v, bar(Smem::v_full + vs), 0, h, i * kStep, r, b);
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const int channel_steps = (P.dim + 15) / 16;
      const uint64_t qdesc = k_major(smem_base + Smem::q);
      bool ok = mbar_wait(bar(Smem::q_full), 0, abort_flag);
      auto issue_scores = [&](int i) {
        ok = mbar_wait(bar(Smem::k_full + i % 3), (i / 3) & 1, abort_flag);
        if (!ok) return;
        tc_fence_after_sync();
        score_product(tmem_base + (i & 1) * kStep, qdesc, k_major(smem_base + Smem::k + (i % 3) * kColTile), channel_steps);
        mma_commit(bar(Smem::s_full + (i & 1)));
        mma_commit(bar(Smem::k_empty + i % 3));
      };
      if (ok) issue_scores(0);
      if (ok && steps > 1) issue_scores(1);
      for (int i = 0; i < steps && ok; ++i) {
        ok = mbar_wait(bar(Smem::v_full + (i & 1)), (i >> 1) & 1, abort_flag);
        if (ok) ok = mbar_wait(bar(Smem::p_full + (i & 1)), (i >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        sum_product(tmem_base + kOCol, tmem_base + (i & 1) * kStep, k_major(smem_base + Smem::v + (i & 1) * kColTile), i == 0);
        mma_commit(bar(Smem::pv_done + (i & 1)));
        mma_commit(bar(Smem::v_empty + (i & 1)));
        if (i + 2 < steps) {  // their columns hold the probabilities that this product reads
          ok = mbar_wait(bar(Smem::pv_done + (i & 1)), (i >> 1) & 1, abort_flag);
          if (ok) issue_scores(i + 2);
        }
      }
    }
  } else {
    const int t = tid;
    const uint32_t lanes = tmem_base + (uint32_t(warp * 32) << 16);
    const f32x2 scale2 = pack2(P.scale, P.scale), log2e2 = pack2(kLog2e, kLog2e);
    // The reference of the softmax rises only when a step's largest logit passes it by `kSlack`: probabilities stay below 2^12 and
    // keep their digits (the split is one of floating-point numbers), and the output is seldom rescaled.
    constexpr float kSlack = 8.f;
    float ref = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int i = 0; i < steps && ok; ++i) {
      const uint32_t s_at = lanes + (i & 1) * kStep;
      if (HAS_BIAS) ok = mbar_wait(bar(Smem::v_full + (i & 1)), (i >> 1) & 1, abort_flag);
      if (ok) ok = mbar_wait(bar(Smem::s_full + (i & 1)), (i >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      f32x2 x[kStep / 2];
      {
        uint32_t s[2][32];
        tmem_ld32(s_at, s[0]);
        tmem_ld32(s_at + 32, s[1]);
        uint4 words[8];
        if (HAS_BIAS) {
          const uint32_t row = smem_base + Smem::bias + (i & 1) * kBiasTile + t * 128 + ((t & 7) << 4);
#pragma unroll
          for (int c = 0; c < 8; ++c) words[c] = lds_v4_at(row ^ uint32_t(c << 4));
        }
        tmem_wait_ld();
        tmem_loaded(s[0]);
        tmem_loaded(s[1]);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t w[4] = {words[c].x, words[c].y, words[c].z, words[c].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int n = 4 * c + e;
            const f32x2 s2 = pack2(__uint_as_float(s[n >> 4][2 * n & 31]), __uint_as_float(s[n >> 4][(2 * n & 31) + 1]));
            x[n] = HAS_BIAS ? fma2(s2, scale2, Half::widen(w[e])) : mul2(s2, scale2);
          }
        }
      }
      if (HAS_BIAS) mbar_arrive_warp(bar(Smem::v_empty + (i & 1)));
      if (i == steps - 1 && P.cols % kStep != 0) {
#pragma unroll
        for (int n = 0; n < kStep / 2; ++n) {
          if (i * kStep + 2 * n >= P.cols) x[n].x = -INFINITY;
          if (i * kStep + 2 * n + 1 >= P.cols) x[n].y = -INFINITY;
        }
      }
      float peaks[4] = {x[0].x, x[1].x, x[2].x, x[3].x};
#pragma unroll
      for (int n = 0; n < kStep / 2; ++n) peaks[n & 3] = max3(peaks[n & 3], x[n].x, x[n].y);
      const float peak = fmaxf(max3(peaks[0], peaks[1], peaks[2]), peaks[3]);
      const bool raised = peak > ref + kSlack || (ref == -INFINITY && peak > ref);
      if (i > 0 && __any_sync(0xffffffffu, raised)) {
        const float shrink = raised ? ex2((ref - peak) * kLog2e) : 1.f;  // 0 for a row without a reference so far
        l_run *= shrink;
        ok = mbar_wait(bar(Smem::pv_done + ((i - 1) & 1)), ((i - 1) >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < kDim; c += 32) {
          uint32_t acc[32];
          tmem_ld32(lanes + kOCol + c, acc);
          tmem_wait_ld();
          tmem_loaded(acc);
#pragma unroll
          for (int n = 0; n < 32; ++n) acc[n] = __float_as_uint(__uint_as_float(acc[n]) * shrink);
          tmem_st32(lanes + kOCol + c, acc);
        }
      }
      if (raised) ref = peak;
      const float shift = ref == -INFINITY ? 0.f : -ref;
      const f32x2 shift2 = pack2(shift, shift);
      f32x2 sums[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        f32x2 p[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          const f32x2 y = mul2(add2(x[8 * c + n], shift2), log2e2);
          p[n] = pack2(ex2(y.x), ex2(y.y));
          sums[n & 1] = add2(sums[n & 1], p[n]);
        }
        uint32_t words[16];
        split16(p, words);
        tmem_st16(s_at + c * 16, words);
      }
      const f32x2 sum = add2(sums[0], sums[1]);
      l_run += sum.x + sum.y;
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive_warp(bar(Smem::p_full + (i & 1)));
    }
    if (ok) ok = mbar_wait(bar(Smem::pv_done + ((steps - 1) & 1)), ((steps - 1) >> 1) & 1, abort_flag);
    if (ok) {
      tc_fence_after_sync();
      const int query = q0 + t;
      const bool some = l_run > 0.f || l_run != l_run;
      const float inv = some ? 1.f / l_run : 0.f;
#pragma unroll 1
      for (int c = 0; c < P.dim; c += 32) {
        uint32_t acc[32];
        tmem_ld32(lanes + kOCol + c, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
        if (query < P.cols) store_channels(P.out, P.dim, b, r, h, query, c, acc, inv);
      }
      if (P.lse && query < P.cols)
        P.lse[((int64_t(b) * P.rows + r) * P.heads + h) * P.cols + query] = some ? ref + lg2(l_run) * kLn2 : 0.f;
    }
  }
  teardown(abort_flag, tmem_base, 5, kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// reverse
// ---------------------------------------------------------------------------------------------
// Eight element-wise warps: two warpgroups whose threads own the same 128 rows, 32 of a step's 64 columns each.
constexpr int kWideElemWarps = 8, kWideProducer = 8, kWideIssuer = 9, kWideBwdThreads = 320;
struct WideBwdSmem {
  // dK/dV and dQ: two row operands, then two stages of two column operands and a bias tile
  static constexpr int rows = 0;
  static constexpr int stages = 2 * kRowTile, stage = 2 * kColTile + kBiasTile;
  static constexpr int stats = stages + 2 * stage;  // [2][2][64] f32: -lse and -delta of a step's queries (dK/dV)
  // bias gradient: two stages of Q, dO (128 rows) and K, V (64 rows)
  static constexpr int tile_stage = 2 * kRowTile + 2 * kColTile;
  static constexpr int bars = (stats + 1024 > 2 * tile_stage ? stats + 1024 : 2 * tile_stage);
  static constexpr int rows_full = 0;
  static constexpr int stage_full = 1, stage_empty = 3;  // [2]
  static constexpr int scores_full = 5, scores_taken = 7;  // [2]
  static constexpr int sums_done = 9;  // [2] by step, for the same reason as the forward kernel's pv_done
  static constexpr int num_bars = 11;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int failed = abort_flag + 4;   // a kernel before this one has given up a wait
  static constexpr int bytes = failed + 4 + 1024;
};
static_assert(WideBwdSmem::bytes <= 113 * 1024, "two reverse CTAs must fit in one SM's shared memory");
enum WideKind { kKeys, kQueries, kBias };

// dK and dV of 128 keys, or dQ of 128 queries.
template <bool HAS_BIAS, WideKind KIND>
__device__ __forceinline__ void wide_rows(const WideParams& P, uint32_t smem_base, uint8_t* smem_gen, volatile int* abort_flag, uint32_t tmem_base,
                                          int tid, int warp, int lane, int idx) {
  using Smem = WideBwdSmem;
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int row0 = idx % P.row_tiles * kTile;
  idx /= P.row_tiles;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int r = idx % P.rows, b = idx / P.rows;
  const int steps = P.steps;
  const int64_t stat0 = ((int64_t(b) * P.rows + r) * P.heads + h) * P.cols;
  // scores | dP | dK | dV; with queries as rows, which leave the scores' columns alone: scores | dP | dQ | dP of odd steps
  constexpr int kSCol = 0, kAcc0 = 2 * kStep, kAcc1 = 2 * kStep + kDim;
  auto d_col = [](int i) { return KIND == kKeys || (i & 1) == 0 ? kStep : 3 * kStep; };
  auto column_tile = [&](int i, int which) { return smem_base + Smem::stages + (i & 1) * Smem::stage + which * kColTile; };
  auto bias_tile = [&](int i) { return column_tile(i, 2); };

  if (warp == kWideProducer) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(bar(Smem::rows_full), 2 * kRowTile);
      tma_load_5d(smem_base + Smem::rows, KIND == kKeys ? &P.key0 : &P.row0, bar(Smem::rows_full), 0, h, row0, r, b);
      tma_load_5d(smem_base + Smem::rows + kRowTile, KIND == kKeys ? &P.key1 : &P.row1, bar(Smem::rows_full), 0, h, row0, r, b);
      for (int i = 0; i < steps && ok; ++i) {
        const int full = Smem::stage_full + (i & 1);
        if (i >= 2) ok = mbar_wait(bar(Smem::stage_empty + (i & 1)), (i / 2 - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(full), 2 * kColTile + (HAS_BIAS ? kBiasTile : 0));
        tma_load_5d(column_tile(i, 0), KIND == kKeys ? &P.col_q : &P.col_k, bar(full), 0, h, i * kStep, r, b);
        tma_load_5d(column_tile(i, 1), KIND == kKeys ? &P.col_d : &P.col_v, bar(full), 0, h, i * kStep, r, b);
        if (HAS_BIAS) {
          const int group = P.bias_groups == 1 ? 0 : r;
          if (KIND == kKeys) tma_load_5d(bias_tile(i), &P.bias_t, bar(full), row0, i * kStep, h, group, b);
          else tma_load_5d(bias_tile(i), &P.bias, bar(full), i * kStep, row0, h, group, b);
        }
      }
    }
  } else if (warp == kWideIssuer) {
    if (lane == 0) {
      const int channel_steps = (P.dim + 15) / 16;
      const uint64_t a0 = k_major(smem_base + Smem::rows), a1 = k_major(smem_base + Smem::rows + kRowTile);
      bool ok = mbar_wait(bar(Smem::rows_full), 0, abort_flag);
      auto issue_scores = [&](int i) {
        ok = mbar_wait(bar(Smem::stage_full + (i & 1)), (i >> 1) & 1, abort_flag);
        // the columns hold what the sums of an earlier step read
        const int before = KIND == kKeys ? i - 1 : i - 2;
        if (ok && before >= 0) ok = mbar_wait(bar(Smem::sums_done + (before & 1)), (before >> 1) & 1, abort_flag);
        if (!ok) return;
        tc_fence_after_sync();
        score_product(tmem_base + kSCol, a0, k_major(column_tile(i, 0)), channel_steps);
        score_product(tmem_base + d_col(i), a1, k_major(column_tile(i, 1)), channel_steps);
        mma_commit(bar(Smem::scores_full));
      };
      if (ok) issue_scores(0);
      for (int i = 0; i < steps && ok; ++i) {
        ok = mbar_wait(bar(Smem::scores_taken), i & 1, abort_flag);
        if (!ok) break;
        if (KIND == kQueries && i + 1 < steps) issue_scores(i + 1);  // the element-wise warps wait for these
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t b0 = k_major(column_tile(i, 0)), b1 = k_major(column_tile(i, 1));
        if (KIND == kKeys) sum_product(tmem_base + kAcc1, tmem_base + kSCol, b1, i == 0);  // dV += P^T dO
        sum_product(tmem_base + kAcc0, tmem_base + d_col(i), b0, i == 0);                  // dK += dS^T Q, dQ += dS K
        mma_commit(bar(Smem::sums_done + (i & 1)));
        mma_commit(bar(Smem::stage_empty + (i & 1)));
        if (KIND == kKeys && i + 1 < steps) issue_scores(i + 1);
      }
    }
  } else if (warp < kWideElemWarps) {
    const int wg = warp >> 2, t = tid & (kTile - 1), at = row0 + t;
    const uint32_t lanes = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const f32x2 scale2 = pack2(P.scale, P.scale);
    float norm = 0.f, neg_delta = 0.f, fetched = 0.f;
    float* stats = reinterpret_cast<float*>(smem_gen + Smem::stats);
    auto fetch = [&](int i) {  // threads 0-63: -lse of the step's queries, 64-127: -delta
      const int q = i * kStep + (tid & 63);
      if (tid < 64) fetched = q < P.cols ? -ldg_f32_here(P.lse + stat0 + q) : -INFINITY;
      else if (tid < 128) fetched = q < P.cols ? -ldg_f32_here(P.delta + stat0 + q) : 0.f;
    };
    if (KIND == kKeys) {
      fetch(0);
    } else {
      norm = at < P.cols ? -P.lse[stat0 + at] : -INFINITY;
      neg_delta = at < P.cols ? -P.delta[stat0 + at] : 0.f;
    }
    bool ok = true;
    for (int i = 0; i < steps && ok; ++i) {
      const float* now = stats + (i & 1) * 128;
      if (KIND == kKeys) {
        if (tid < 128) stats[(i & 1) * 128 + tid] = fetched;
        if (i + 1 < steps) fetch(i + 1);
        named_barrier_sync(1, kWideElemWarps * 32);
      }
      if (HAS_BIAS) ok = mbar_wait(bar(Smem::stage_full + (i & 1)), (i >> 1) & 1, abort_flag);
      if (ok) ok = mbar_wait(bar(Smem::scores_full), i & 1, abort_flag);
      // (every warp passes the barrier above as often as the others, whatever became of its waits)
      if (ok) tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 2 && ok; ++c) {
        const int col = wg * 32 + c * 16;  // sixteen columns of the step
        uint32_t s[16], d[16];
        tmem_ld16(lanes + kSCol + col, s);
        tmem_ld16(lanes + d_col(i) + col, d);
        f32x2 add[8];
        if (HAS_BIAS && KIND == kQueries) {
          const uint32_t row = bias_tile(i) + t * 128 + ((t & 7) << 4);
          const uint4 lo = lds_v4_at(row ^ uint32_t((col / 8) << 4)), hi = lds_v4_at(row ^ uint32_t((col / 8 + 1) << 4));
          const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
          for (int n = 0; n < 8; ++n) add[n] = Half::widen(w[n]);
        } else {
#pragma unroll
          for (int n = 0; n < 8; ++n) add[n] = pack2(0.f, 0.f);
        }
        // kKeys: queries are the bias tile's rows, and the threads of a warp read neighbouring keys of one query
        const uint16_t* key = reinterpret_cast<const uint16_t*>(smem_gen + (bias_tile(i) - smem_base)) + col * kTile + t;
        tmem_wait_ld();
        tmem_loaded(s);
        tmem_loaded(d);
        f32x2 p[8], ds[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          f32x2 norm2 = pack2(norm, norm), delta2 = pack2(neg_delta, neg_delta);
          if (KIND == kKeys) {
            norm2 = *reinterpret_cast<const float2*>(now + col + 2 * n);
            delta2 = *reinterpret_cast<const float2*>(now + 64 + col + 2 * n);
            if (HAS_BIAS) add[n] = pack2(__uint_as_float(uint32_t(key[2 * n * kTile]) << 16), __uint_as_float(uint32_t(key[(2 * n + 1) * kTile]) << 16));
          }
          p[n] = probability(pack2(__uint_as_float(s[2 * n]), __uint_as_float(s[2 * n + 1])), scale2, add[n], norm2);
          ds[n] = mul2(p[n], add2(pack2(__uint_as_float(d[2 * n]), __uint_as_float(d[2 * n + 1])), delta2));
        }
        if (KIND == kQueries && i == steps - 1 && P.cols % kStep != 0) {
#pragma unroll
          for (int n = 0; n < 8; ++n) {  // no such keys
            if (i * kStep + col + 2 * n >= P.cols) ds[n].x = 0.f;
            if (i * kStep + col + 2 * n + 1 >= P.cols) ds[n].y = 0.f;
          }
        }
        uint32_t words[16];
        if (KIND == kKeys) {
          split16(p, words);
          tmem_st16(lanes + kSCol + col, words);
        }
        split16(ds, words);
        tmem_st16(lanes + d_col(i) + col, words);
      }
      if (ok) {
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive_warp(bar(Smem::scores_taken));
      }
      if (KIND == kKeys && !ok) {  // the others of the CTA still meet at the barrier
        for (int rest = i + 1; rest < steps; ++rest) named_barrier_sync(1, kWideElemWarps * 32);
      }
    }
    if (ok) ok = mbar_wait(bar(Smem::sums_done + ((steps - 1) & 1)), ((steps - 1) >> 1) & 1, abort_flag);
    if (ok) {
      tc_fence_after_sync();
      if (KIND == kKeys) {  // a warpgroup per gradient
        const oops_ta_pair& to = wg == 0 ? P.dk : P.dv;
#pragma unroll 1
        for (int c = 0; c < P.dim; c += 32) {
          uint32_t acc[32];
          tmem_ld32(lanes + (wg == 0 ? kAcc0 : kAcc1) + c, acc);
          tmem_wait_ld();
          tmem_loaded(acc);
          if (at < P.cols && to.ptr) store_channels(to, P.dim, b, r, h, at, c, acc, wg == 0 ? P.scale : 1.f);
        }
      } else if (wg * 32 < P.dim) {
        uint32_t acc[32];
        tmem_ld32(lanes + kAcc0 + wg * 32, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
        if (at < P.cols) store_channels(P.dq, P.dim, b, r, h, at, wg * 32, acc, P.scale);
      }
    }
  }
}

// A 128 x 64 tile of the row-shared bias gradient: the sum of dS over the part's rows.
__device__ __forceinline__ void wide_bias(const WideParams& P, uint32_t smem_base, uint8_t* smem_gen, volatile int* abort_flag, uint32_t tmem_base,
                                          int tid, int warp, int lane, int idx) {
  using Smem = WideBwdSmem;
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int k0 = idx % P.steps * kStep;
  idx /= P.steps;
  const int q0 = idx % P.row_tiles * kTile;
  idx /= P.row_tiles;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int b = idx % P.batch, part = idx / P.batch;
  const int first = part * P.rows_per_part, count = min(P.rows, first + P.rows_per_part) - first;
  auto tile = [&](int i, int offset) { return smem_base + (i & 1) * Smem::tile_stage + offset; };
  constexpr int kDo = kRowTile, kKey = 2 * kRowTile, kVal = 2 * kRowTile + kColTile;

  if (warp == kWideProducer) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < count && ok; ++i) {
        const int full = Smem::stage_full + (i & 1), r = first + i;
        if (i >= 2) ok = mbar_wait(bar(Smem::stage_empty + (i & 1)), (i / 2 - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(full), Smem::tile_stage);
        tma_load_5d(tile(i, 0), &P.row0, bar(full), 0, h, q0, r, b);
        tma_load_5d(tile(i, kKey), &P.col_k, bar(full), 0, h, k0, r, b);
        tma_load_5d(tile(i, kDo), &P.row1, bar(full), 0, h, q0, r, b);
        tma_load_5d(tile(i, kVal), &P.col_v, bar(full), 0, h, k0, r, b);
      }
    }
  } else if (warp == kWideIssuer) {
    if (lane == 0) {
      const int channel_steps = (P.dim + 15) / 16;
      bool ok = true;
      for (int i = 0; i < count && ok; ++i) {
        ok = mbar_wait(bar(Smem::stage_full + (i & 1)), (i >> 1) & 1, abort_flag);
        if (ok && i >= 2) ok = mbar_wait(bar(Smem::scores_taken + (i & 1)), ((i >> 1) - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t at = tmem_base + (i & 1) * 2 * kStep;
        score_product(at, k_major(tile(i, 0)), k_major(tile(i, kKey)), channel_steps);
        score_product(at + kStep, k_major(tile(i, kDo)), k_major(tile(i, kVal)), channel_steps);
        mma_commit(bar(Smem::scores_full + (i & 1)));
        mma_commit(bar(Smem::stage_empty + (i & 1)));
      }
    }
  } else if (warp < kWideElemWarps) {
    const int wg = warp >> 2, t = tid & (kTile - 1), query = q0 + t, key0 = k0 + wg * 32;
    const uint32_t lanes = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const f32x2 scale2 = pack2(P.scale, P.scale);
    uint32_t words[16];  // the thread's 32 bias values
    const uint16_t* from = reinterpret_cast<const uint16_t*>(P.bias_ptr) + b * P.b_sb + h * P.b_sh + int64_t(query) * P.b_sq + key0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (query < P.cols && key0 + 8 * c + 8 <= P.cols) {
        v = *reinterpret_cast<const uint4*>(from + 8 * c);
      } else if (query < P.cols) {
        uint16_t e[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) e[n] = key0 + 8 * c + n < P.cols ? from[8 * c + n] : uint16_t(0);
        v = make_uint4(e[0] | uint32_t(e[1]) << 16, e[2] | uint32_t(e[3]) << 16, e[4] | uint32_t(e[5]) << 16, e[6] | uint32_t(e[7]) << 16);
      }
      words[4 * c] = v.x;
      words[4 * c + 1] = v.y;
      words[4 * c + 2] = v.z;
      words[4 * c + 3] = v.w;
    }
    f32x2 sums[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) sums[n] = pack2(0.f, 0.f);
    float norm, neg_delta;
    auto fetch = [&](int i) {
      norm = -INFINITY;
      neg_delta = 0.f;
      if (i < count && query < P.cols) {
        const int64_t stat = ((int64_t(b) * P.rows + first + i) * P.heads + h) * P.cols + query;
        norm = -ldg_f32_here(P.lse + stat);
        neg_delta = -ldg_f32_here(P.delta + stat);
      }
    };
    fetch(0);
    bool ok = true;
    for (int i = 0; i < count; ++i) {
      const f32x2 norm2 = pack2(norm, norm), delta2 = pack2(neg_delta, neg_delta);
      fetch(i + 1);
      ok = mbar_wait(bar(Smem::scores_full + (i & 1)), (i >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t at = lanes + (i & 1) * 2 * kStep + wg * 32;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t s[8], d[8];
        tmem_ld8(at + c * 8, s);
        tmem_ld8(at + kStep + c * 8, d);
        tmem_wait_ld();
        tmem_loaded(s);
        tmem_loaded(d);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const f32x2 p = probability(pack2(__uint_as_float(s[2 * n]), __uint_as_float(s[2 * n + 1])), scale2, Half::widen(words[4 * c + n]), norm2);
          sums[4 * c + n] = fma2(p, add2(pack2(__uint_as_float(d[2 * n]), __uint_as_float(d[2 * n + 1])), delta2), sums[4 * c + n]);
        }
      }
      tc_fence_before_sync();
      mbar_arrive_warp(bar(Smem::scores_taken + (i & 1)));
    }
    if (!ok) return;
    const int width = min(32, P.cols - key0);
    auto value = [&](int n) { return n & 1 ? sums[n >> 1].y : sums[n >> 1].x; };
    const bool split = P.num_parts > 1, f32 = split || P.dbias_f32;
    const int64_t sq = split ? P.cols : P.db_sq, sk = split ? 1 : P.db_sk;
    const int64_t to = (split ? ((int64_t(part) * P.batch + b) * P.heads + h) * P.cols * P.cols : b * P.db_sb + h * P.db_sh) + int64_t(query) * sq + key0 * sk;
    float* row32 = (split ? P.parts : reinterpret_cast<float*>(P.dbias)) + to;
    __nv_bfloat16* row16 = reinterpret_cast<__nv_bfloat16*>(P.dbias) + to;
    if (P.store_words && width == 32) {  // every row of the gradient starts on a 16-byte word
      if (query >= P.cols) return;
      if (f32) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          reinterpret_cast<float4*>(row32)[c] = make_float4(value(4 * c), value(4 * c + 1), value(4 * c + 2), value(4 * c + 3));
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          reinterpret_cast<uint4*>(row16)[c] = make_uint4(Half::pack(value(8 * c), value(8 * c + 1)), Half::pack(value(8 * c + 2), value(8 * c + 3)),
                                                          Half::pack(value(8 * c + 4), value(8 * c + 5)), Half::pack(value(8 * c + 6), value(8 * c + 7)));
      }
      return;
    }
    // Otherwise the warp's 32 x 32 tile goes through shared memory, whose operands every product has read by now, so that a
    // store covers 32 neighbouring keys of one query.
    float* tile32 = reinterpret_cast<float*>(smem_gen) + warp * 32 * 33;
#pragma unroll
    for (int n = 0; n < 32; ++n) tile32[lane * 33 + n] = value(n);
    __syncwarp();
    if (lane >= width) return;
    const int rows = min(32, P.cols - (query - lane));
    const int64_t first_row = to - int64_t(lane) * sq + lane * sk;
    for (int n = 0; n < rows; ++n) {
      const float v = tile32[n * 33 + lane];
      const int64_t at = first_row + int64_t(n) * sq;
      if (f32) (split ? P.parts : reinterpret_cast<float*>(P.dbias))[at] = v;
      else reinterpret_cast<__nv_bfloat16*>(P.dbias)[at] = __float2bfloat16_rn(v);
    }
  }
}

template <bool HAS_BIAS>
__global__ void __launch_bounds__(kWideBwdThreads, 2) ta_wide_bwd_kernel(const __grid_constant__ WideParams P) {
  using Smem = WideBwdSmem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Smem::abort_flag);
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == kWideProducer) {
    const bool failed = device_failed();  // (looked at beside the other preparations)
    if (lane < Smem::num_bars) mbar_init(bar(lane), lane >= Smem::scores_taken && lane < Smem::sums_done ? kWideElemWarps : 1);
    fence_barrier_init();
    if (lane == 0) {
      *abort_flag = 0;
      *reinterpret_cast<volatile int*>(smem_gen + Smem::failed) = failed ? 1 : 0;
    }
  }
  if (warp == kWideIssuer) {
    tmem_alloc(smem_base + Smem::tmem_slot, kTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_gen + Smem::tmem_slot);
  const int idx = int(blockIdx.x);
  if (*reinterpret_cast<volatile int*>(smem_gen + Smem::failed) != 0) {
    // nothing has been requested: on to the end
  } else if (idx < P.dkv_ctas) {
    wide_rows<HAS_BIAS, kKeys>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, idx);
  } else if (idx < P.dkv_ctas + P.dq_ctas) {
    wide_rows<HAS_BIAS, kQueries>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, idx - P.dkv_ctas);
  } else if (HAS_BIAS) {
    wide_bias(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, idx - P.dkv_ctas - P.dq_ctas);
  }
  teardown(abort_flag, tmem_base, kWideIssuer, kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
int encode_rows(CUtensorMap* map, const oops_ta_problem& p, const oops_ta_pair& t, uint32_t box_cols, const char* what) {
  const uint64_t dims[5] = {uint64_t(p.head_dim), uint64_t(p.heads), uint64_t(p.cols), uint64_t(p.rows), uint64_t(p.batch)};
  const int64_t strides[4] = {t.sh, t.sc, t.sr, t.sb};
  const uint32_t box[5] = {kDim, 1, box_cols, 1, 1};
  return encode_map(map, p.dtype, t.ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, what);
}

// What a tensor map holds: strides below 2^40 bytes.
bool mappable(const oops_ta_pair& t) { return std::max(std::max(t.sb, t.sr), std::max(t.sc, t.sh)) < int64_t(1) << 39; }

bool stored_whole(const oops_ta_pair& t) {
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 8 == 0 && t.sr % 8 == 0 && t.sc % 8 == 0 && t.sh % 8 == 0;
}

void describe(WideParams& P, const oops_ta_problem& p) {
  P.batch = p.batch;
  P.rows = p.rows;
  P.cols = p.cols;
  P.heads = p.heads;
  P.dim = p.head_dim;
  P.bias_groups = p.bias_groups;
  P.row_tiles = (int)ceil_div(p.cols, kTile);
  P.steps = (int)ceil_div(p.cols, kStep);
  P.scale = p.scale;
}

template <typename Kernel>
int launch(Kernel kernel, const WideParams& P, int64_t grid, int threads, int smem, cudaStream_t stream, const char* what) {
  const int status = reserve_smem(kernel, smem);
  if (status) return status;
  kernel<<<(unsigned)grid, threads, smem, stream>>>(P);
  count_launch();
  return check_launch(what);
}

int64_t row_ctas(const oops_ta_problem& p) { return int64_t(p.batch) * p.rows * p.heads * ceil_div(p.cols, kTile); }

}  // namespace

namespace {

bool served(const oops_ta_problem& p) {
  if (p.dtype != OOPS_TA_BF16 || p.mask || p.head_dim > kDim || p.head_dim % 8 != 0) return false;
  for (const oops_ta_pair* t : {&p.q, &p.k, &p.v})
    if (!pair_ok(*t, p) || !mappable(*t)) return false;
  if (p.bias_groups != 0) {
    if (p.bias_dtype != p.dtype || p.bias_sk != 1 || p.cols == 1 || (reinterpret_cast<uintptr_t>(p.bias) & 15) != 0) return false;
    if (!stride_ok(p.bias_sq, p.cols) || !stride_ok(p.bias_sh, p.heads) || !stride_ok(p.bias_sg, p.bias_groups) || !stride_ok(p.bias_sb, p.batch))
      return false;
    if (!mappable({nullptr, p.bias_sb, p.bias_sg, p.bias_sh, p.bias_sq})) return false;
  }
  return row_ctas(p) <= 0x7fffffffll;
}

}  // namespace

static int padded_dim(const oops_ta_problem& p) { return (int)ceil_div(p.head_dim, 16) * 16; }

// A call of few columns and channels ends before the barriers, tensor memory and copies of these kernels are set up: 64 problems of 64
// columns and 16 channels take 3.3 us at register level and 4.3 here, 128 columns and 24 channels 5.1 and 5.5; with 48
// channels it is 6.6 and 5.8, and 8 problems of 128 columns and 64 channels take 7.0 and 5.3.  Up to 16 channels on half of the SMs it
// is longer columns that pay (8 problems of 300 columns: 7.9 and 8.2, of 384: 9.1 and 8.7; 384 problems of 300: 39 and 34).
bool wide_forward_applies(const oops_ta_problem& p, const oops_ta_pair& out) {
  const int channels = padded_dim(p), least = channels == 16 && row_ctas(p) <= 74 ? 383 * 16 : 4096;
  return int64_t(p.cols) * channels > least && served(p) && stored_whole(out);
}

int wide_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream) {
  WideParams P{};
  describe(P, p);
  int status = encode_rows(&P.row0, p, p.q, kTile, "query");
  if (!status) status = encode_rows(&P.col_k, p, p.k, kStep, "key");
  if (!status) status = encode_rows(&P.col_v, p, p.v, kStep, "value");
  if (!status && p.bias_groups) status = encode_bias(&P.bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
  if (status) return status;
  P.out = out;
  P.lse = lse;
  return p.bias_groups ? launch(ta_wide_fwd_kernel<true>, P, row_ctas(p), kWideFwdThreads, WideFwdSmem::bytes, stream, "wide forward")
                       : launch(ta_wide_fwd_kernel<false>, P, row_ctas(p), kWideFwdThreads, WideFwdSmem::bytes, stream, "wide forward");
}

// Which of the two reverse kernels is the faster one, from 8 to 768 columns in 1, some and many problems (a row and head each), times of the
// register-level kernels first.  Tiles of 128 rows against 64: up to 64 columns half of a tile is empty, from 129 to 192 a quarter, which
// costs more than the tensor pipe saves where there are few channels; and a CTA takes longer to set up than a small call does to end.
//   bias gradient alone     here: 13 / 7 us (8 problems of 64 columns and 64 channels) to 583 / 137 (384 of 768); never slower.
//   up to 64 columns        without a bias gradient here only where 48 or more channels fit one wave (148 problems of 64 columns and 64 channels:
//                           11.5 / 9.6; 4096: 155 / 168, with 16 channels 81 / 134); with one here from 24 channels on (4096 problems: 220 / 209; 16
//                           channels 173 / 188, 8 problems of them 9.1 / 7.4).
//   more, 16 channels       129 to 192 columns at register level (1024 problems of 160: 108 / 122 us), but for many problems of more than 8 channels with a
//                           bias gradient (162 / 154; 8 channels 161 / 167; 48 problems of 16 19 / 21); else by problems and columns (8 problems of 256:
//                           11.8 / 12.7, with the bias gradient 12.2 / 12.7, of 384 18.1 / 17.1; 28 of 300, queries alone: 11.6 / 12.3; 1024 of 256: 177 / 154
//                           and 265 / 206).
//   more, 32 channels       on a quarter of the SMs without a bias gradient at register level below 256 columns (8 of 192: 11.3 / 12.0).
//   more, 48 channels       here (8 problems of 65 columns: 10.9 / 10.1; 1024 of 256: 331 / 193).
static bool wide_backward_pays(const oops_ta_problem& p, const oops_ta_grads& g) {
  const bool keys = g.dk.ptr || g.dv.ptr, queries = g.dq.ptr != nullptr;
  if (!keys && !queries) return true;
  const int channels = padded_dim(p);
  const int64_t problems = row_ctas(p), ctas = problems * (int(keys) + int(queries));
  if (p.cols <= 64) return g.dbias ? channels >= 32 || problems <= 16 : channels >= 48 && ctas <= 296;
  if (channels >= 48) return true;
  if (channels == 32) return g.dbias || ctas > 37 || p.cols >= 256;
  if (p.cols > kTile && p.cols <= 192) return g.dbias && p.head_dim > 8 && problems > 296;
  return g.dbias ? problems > 32 || p.cols >= 384 : problems > (keys && queries ? 37 : 148) || p.cols >= 1024;
}

bool wide_backward_applies(const oops_ta_problem& p, const oops_ta_pair& dout, const oops_ta_grads& g) {
  if (p.bias_groups > 1 && g.dbias) return false;
  if (!wide_backward_pays(p, g) || !served(p) || !pair_ok(dout, p) || !mappable(dout)) return false;
  for (const oops_ta_pair* t : {&g.dq, &g.dk, &g.dv})
    if (t->ptr && !stored_whole(*t)) return false;
  const int64_t tiles = int64_t(p.batch) * p.heads * ceil_div(p.cols, kTile) * ceil_div(p.cols, kStep);
  return 2 * row_ctas(p) + 16 * tiles <= 0x7fffffffll;
}

int wide_backward(const oops_ta_problem& p, const oops_ta_pair& dout, const float* lse, const float* delta, const oops_ta_grads& g, int num_parts,
                  float* parts, cudaStream_t stream) {
  WideParams P{};
  describe(P, p);
  int status = encode_rows(&P.row0, p, p.q, kTile, "query");
  if (!status) status = encode_rows(&P.row1, p, dout, kTile, "dout");
  if (!status) status = encode_rows(&P.key0, p, p.k, kTile, "key");
  if (!status) status = encode_rows(&P.key1, p, p.v, kTile, "value");
  if (!status) status = encode_rows(&P.col_q, p, p.q, kStep, "query");
  if (!status) status = encode_rows(&P.col_d, p, dout, kStep, "dout");
  if (!status) status = encode_rows(&P.col_k, p, p.k, kStep, "key");
  if (!status) status = encode_rows(&P.col_v, p, p.v, kStep, "value");
  if (!status && p.bias_groups) {
    status = encode_bias(&P.bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
    const uint64_t dims[5] = {uint64_t(p.cols), uint64_t(p.cols), uint64_t(p.heads), uint64_t(p.bias_groups), uint64_t(p.batch)};
    const int64_t strides[4] = {p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb};
    const uint32_t box[5] = {kTile, kStep, 1, 1, 1};
    if (!status) status = encode_map(&P.bias_t, p.dtype, p.bias, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "bias columns");
  }
  if (status) return status;
  P.dq = g.dq;
  P.dk = g.dk;
  P.dv = g.dv;
  P.lse = const_cast<float*>(lse);
  P.delta = delta;
  P.bias_ptr = p.bias;
  P.b_sb = p.bias_sb;
  P.b_sh = p.bias_sh;
  P.b_sq = p.bias_sq;
  P.dkv_ctas = g.dk.ptr || g.dv.ptr ? (int)row_ctas(p) : 0;
  P.dq_ctas = g.dq.ptr ? (int)row_ctas(p) : 0;
  int64_t grid = int64_t(P.dkv_ctas) + P.dq_ctas;
  if (g.dbias) {
    P.dbias = g.dbias;
    P.parts = parts;
    P.db_sb = g.dbias_sb;
    P.db_sh = g.dbias_sh;
    P.db_sq = g.dbias_sq;
    P.db_sk = g.dbias_sk;
    P.dbias_f32 = (p.flags & OOPS_TA_FLAG_DBIAS_F32) != 0;
    P.num_parts = num_parts;
    P.rows_per_part = (int)ceil_div(p.rows, num_parts);
    P.store_words = num_parts > 1 ? p.cols % 4 == 0 && (reinterpret_cast<uintptr_t>(parts) & 15) == 0
                                  : g.dbias_sk == 1 && (reinterpret_cast<uintptr_t>(g.dbias) & 15) == 0 && g.dbias_sb % 8 == 0 && g.dbias_sh % 8 == 0 &&
                                        g.dbias_sq % 8 == 0;
    grid += int64_t(num_parts) * p.batch * p.heads * P.row_tiles * P.steps;
  }
  if (grid == 0) return OOPS_TA_OK;
  return p.bias_groups ? launch(ta_wide_bwd_kernel<true>, P, grid, kWideBwdThreads, WideBwdSmem::bytes, stream, "wide backward")
                       : launch(ta_wide_bwd_kernel<false>, P, grid, kWideBwdThreads, WideBwdSmem::bytes, stream, "wide backward");
}

int wide_device_status(int reset) { return read_tu_device_status(reset); }

}  // namespace oops_ta
