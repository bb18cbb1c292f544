// tcgen05 / TMEM / TMA triangle-attention kernels for sm_100a (f16 and bf16, head_dim 32).
//
// Forward (replaces the reference's Triton `_attend`, oops/attention/triangle/triton/kernel.py:150-262):
// a CTA works on two 128-query tiles.  With a row-shared bias (or none) the tiles are the same queries of two neighbouring
// pair rows, which read one bias tile; with a per-row bias they are neighbouring query tiles of one row, which read one
// K/V stream.  A producer warp streams 64-key K/V tiles and 128 x 64 bias tiles into shared memory with TMA; a thread per
// tile issues tcgen05.mma for S = Q K^T (accumulator in tensor memory) and O += P V (P read back from tensor memory,
// V from shared memory); one softmax warpgroup per tile (a thread owns a query) turns S into P.
//
// The softmax has no row maximum in its steady state.  The maximum of a row's first step is its reference (that probability
// is then 1, which 16 bits hold exactly; a reference from fewer columns left every large one rounded, and short rows 2 to 5 %
// further from the exact result); later steps take 2^(x - reference) as they come, 16 columns at a time, and look at their sum only: 2^10
// or more in the first 48 columns (or a NaN), or a logit of 10 or more in the last 16, sends the warp back over the step, which still
// stands in tensor memory, to raise the reference and rescale the accumulators.  Probabilities therefore stay below 2^10, inside the
// f32, bf16 and f16 ranges.  With that look the scores are given back before the exponentials of the last 16 columns, and the next
// score product runs under them (N = 768: 711 -> 683 us, 512: 234 -> 222, 2048: 11.6 -> 11.23 ms; an all-ones mask, 768: 726 -> 702).  A step that
// tests kept bits looks at the sum of all its columns and gives its scores back with its probabilities: there the look at the last logits costs more
// than the lead of the product gives (scattered keys of 768 columns 936 us, without it 924), and a report of its own for the scores 1 %.
// Against a maximum per step this saves the comparisons, and above all the wait: no exponential depended on the last
// score of a step any more, scores need not be held in registers, and an exponential costs 5 instead of 9.5 issue slots.
// What bounds it: the element-wise warps' streams, with the special-function unit (63 %; one ex2 per score at 16 per clock and SM,
// 0.39 of the 0.68 ms at N = 768) and issue slots (60 %) the busiest units.  Eight softmax warps of an SM alone reach 70 to 80 % of what
// sixteen do.  Without a bias the kernel takes 0.57 ms; giving the bias another way did not help: as f32 blocks that tcgen05.cp copies
// into the score accumulators 0.74 ms (a copy of 4 KB holds the tensor queue for some hundred clocks), as f32 in shared memory 0.69;
// nor did exponentials on the FMA pipe (1/8: 0.71, 1/4: 0.74) or logits computed between the exponentials of the columns before
// (0.69).  Hence no tests on kept bits where nothing is dropped: a CTA whose rows keep every key walks a copy
// of the roles without them (N = 768: 757 -> 703 us), and otherwise the steps that every row keeps whole come first, in a
// loop of their own (the order of the keys is free; N = 1024, 1000 kept: 1659 -> 1618 us), and a step that one of two rows
// keeps costs the other a row of zeros (N = 1000, rows that keep alternate blocks of 64 keys: 1966 -> 1466 us).
#include <type_traits>

#include "ta_tensor_common.cuh"

namespace oops_ta {
namespace {

using namespace ptx;

constexpr int kStages = 3;                       // K/V ring depth
constexpr int kKeys = 64;                        // keys per step
constexpr int kQBytes = kTile * kHeadDim * 2;    // 8 KiB: one 128-query Q tile
constexpr int kKvBytes = kKeys * kHeadDim * 2;   // 4 KiB: one K or V step
constexpr int kBiasBytes = kTile * kKeys * 2;    // 16 KiB: one 128 x 64 bias tile (one swizzle-128 box)
constexpr int kFwdThreads = 352;                 // 2 softmax warpgroups + producer warp + 2 MMA warps
constexpr int kFwdTmemCols = 256;                // S 2x64 | P 2x32 | O 2x32; two CTAs share an SM
constexpr int kMaxKeepWords = 512;               // keep-bit table: one bit per key column, cols <= 16384

// ROWS: the two tiles belong to two pair rows (own K/V rings, one bias ring); otherwise to one row (one K/V ring, own
// bias rings).
template <bool ROWS>
struct FwdSmem {
  static constexpr int kv_rings = ROWS ? 2 : 1, bias_rings = ROWS ? 1 : 2;
  static constexpr int q = 0;                                     // [2]
  static constexpr int k = q + 2 * kQBytes;                       // [kv_rings][kStages]
  static constexpr int v = k + kv_rings * kStages * kKvBytes;     // [kv_rings][kStages]
  static constexpr int bias = v + kv_rings * kStages * kKvBytes;  // [bias_rings][2 buffers]
  static constexpr int bars = bias + bias_rings * 2 * kBiasBytes;
  // barrier indices (8 bytes each)
  static constexpr int q_full = 0;                                // [2]
  static constexpr int k_full = q_full + 2;                       // [kv_rings][kStages]
  static constexpr int k_empty = k_full + kv_rings * kStages;
  static constexpr int v_full = k_empty + kv_rings * kStages;
  static constexpr int v_empty = v_full + kv_rings * kStages;
  static constexpr int v_ready = v_empty + kv_rings * kStages;    // rows of dropped keys have been cleared
  static constexpr int bias_full = v_ready + kv_rings * kStages;  // [bias_rings][2 buffers]
  static constexpr int bias_empty = bias_full + bias_rings * 2;
  static constexpr int s_full = bias_empty + bias_rings * 2;      // [2] S of a step is in tensor memory
  static constexpr int p_full = s_full + 2;                       // [2] P is in tensor memory
  static constexpr int s_free = p_full + 2;                       // [2] the scores of a step that gives them back early are in registers
  static constexpr int pv_done = s_free + 2;                      // [2] the latest P V product has completed
  static constexpr int q_empty = pv_done + 2;                     // [2] every score product of an item has completed (PERSIST)
  static constexpr int num_bars = q_empty + 2;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int lost_flag = abort_flag + 4;                // a row of a walk over a closed bias came out as NaN
  static constexpr int drop_flags = lost_flag + 4;               // [8] per-warp: the mask drops a key of this row
  static constexpr int step_count = drop_flags + 32;
  static constexpr int full_count = step_count + 4;
  static constexpr int steps = full_count + 4;                    // [2][256] u16: full steps, other steps with a kept key
  static constexpr int keep = (steps + 1024 + 15) / 16 * 16;       // [kv_rings][kMaxKeepWords] u32
  static constexpr int total = keep + kv_rings * kMaxKeepWords * 4;
  static constexpr int bytes = total + 1024;                      // slack to align the base to 1 KiB
};
static_assert(FwdSmem<true>::bytes <= 113 * 1024 && FwdSmem<false>::bytes <= 113 * 1024,
              "two forward CTAs must fit in one SM's shared memory");

struct FwdParams {
  CUtensorMap map_q, map_k, map_v, map_bias;
  void* out;
  int64_t o_sb, o_sr, o_sc, o_sh;
  float* lse;
  const uint8_t* mask;
  int64_t m_sb, m_sr, m_sc;
  int batch, rows, cols, heads, bias_groups;
  int closed;            // the bias is minus infinity behind a ragged row's end
  Logits logits;         // its operands (a closed bias only)
  int items;             // query items x heads x rows (or pairs of rows) x batch
  int q_items, k_steps;  // query tiles (ROWS) or pairs of query tiles of a row; key steps
  int out_vec16;
  float scale;
  // gated epilogue (GATED instantiations): gated = sigmoid(gate) * out goes to `out`, the ungated values to `plain`
  const void* gate;
  int64_t g_sb, g_sr, g_sc, g_sh;
  void* plain;  // may be null
  int64_t p_sb, p_sr, p_sc, p_sh;
  int gate_vec16, plain_vec16;
};

// What sends a step's warp back for a new reference: the sum of the probabilities of the first 48 columns, or a base-2 logit of the last 16 (whose
// probabilities are not known yet when the scores are given back); in a step with tests the sum of all.  No probability reaches 2^10 then, no step's sum 2^15.
constexpr float kStepSumLimit = 1024.f, kLastColumnsLimit = 10.f;

// Where item `idx` lies: query item fastest, then head, row (or pair of rows), batch.
struct FwdItem {
  int h, r0, b, q0;
};
template <bool ROWS>
__device__ __forceinline__ FwdItem fwd_item(const FwdParams& P, int idx) {
  const int qi = idx % P.q_items;
  idx /= P.q_items;
  const int h = idx % P.heads;
  idx /= P.heads;
  const int row_items = ROWS ? (P.rows + 1) / 2 : P.rows;
  return {h, (idx % row_items) * (ROWS ? 2 : 1), idx / row_items, qi * (ROWS ? kTile : 2 * kTile)};
}

// What the CTA's roles do once its set-up stands.  PLAIN: every key of every row is kept.  `masked`: otherwise the mask drops
// some, and the step list stands.  PERSIST: the CTA goes on to further items, the first step's copies and score products of
// the next one under the last steps and the output of this one; barrier phases count steps across items.
template <typename T, bool HAS_BIAS, bool GATED, bool ROWS, bool PERSIST, bool PLAIN>
__device__ __forceinline__ void fwd_walk(const FwdParams& P, uint32_t smem_base, uint8_t* smem_gen, volatile int* abort_flag,
                                         uint32_t tmem_base, int tid, int warp, int lane, FwdItem at, int n_tiles, bool masked) {
  using Smem = FwdSmem<ROWS>;
  const uint32_t* keep_words = reinterpret_cast<const uint32_t*>(smem_gen + Smem::keep);
  const uint16_t* step_list = reinterpret_cast<const uint16_t*>(smem_gen + Smem::steps);
  const uint32_t* drop_flags = reinterpret_cast<const uint32_t*>(smem_gen + Smem::drop_flags);
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int n_rings = ROWS ? n_tiles : 1;
  const bool listed = !PLAIN && masked;
  // Steps whose scores are given back early: those without tests, but not where the tiles of one row share a list (300 columns, 91 % of the tokens,
  // a bias per row: 104.6 us, with them 108.5).
  constexpr bool kEarly = PLAIN || ROWS;
  // (a last row without a partner is its own partner in a persistent walk, whose barriers count two tiles)
  auto row_of = [&](int w) { return ROWS ? (PERSIST ? min(at.r0 + w, P.rows - 1) : at.r0 + w) : at.r0; };
  auto first_query = [&](int w) { return ROWS ? at.q0 : at.q0 + w * kTile; };
  auto item_there = [&](int item, int turn) { return PERSIST ? item < P.items : turn == 0; };
  const int KS = listed ? *reinterpret_cast<volatile int*>(smem_gen + Smem::step_count) : P.k_steps;
  const int full_steps = PLAIN ? KS : listed ? *reinterpret_cast<volatile int*>(smem_gen + Smem::full_count) : P.cols / kKeys;  // come first; the others test their kept bits
  auto step_at = [&](int i) { return listed ? int(step_list[i < full_steps ? i : 256 + i - full_steps]) : i; };
  // Value rows only need the sign-off handshake when the mask really drops a key of the row.
  auto needs_signoff = [&](int w) {
    bool drops = false;
    if (listed) {
#pragma unroll
      for (int i = 0; i < 8; ++i) drops |= (!ROWS || (i >> 2) == w) && drop_flags[i] != 0;
    }
    return drops;
  };
  // tensor-memory columns
  constexpr int kSCol = 0, kPCol = 2 * kKeys, kOCol = 2 * kKeys + 2 * (kKeys / 2);

  if (warp == 8) {
    // ------------------------------------------------------------------ producer (one thread)
    if (lane == 0) {
      bool ok = true;
      if (KS == 0)  // nobody else waits for the queries: the CTA must not leave before they have landed
        for (int w = 0; w < n_tiles && ok; ++w) ok = mbar_wait(bar(Smem::q_full + w), 0, abort_flag);
      int n = 0;  // steps so far
      for (int item = int(blockIdx.x), turn = 0; ok && item_there(item, turn); item += int(gridDim.x), ++turn) {
        if (PERSIST && turn > 0) {
          at = fwd_item<ROWS>(P, item);
          for (int w = 0; w < n_tiles && ok; ++w) {
            ok = mbar_wait(bar(Smem::q_empty + w), (turn - 1) & 1, abort_flag);
            if (!ok) break;
            mbar_expect_tx(bar(Smem::q_full + w), kQBytes);
            tma_load_5d(smem_base + Smem::q + w * kQBytes, &P.map_q, bar(Smem::q_full + w), 0, at.h, first_query(w), row_of(w), at.b);
          }
        }
        for (int i = 0; i < KS && ok; ++i, ++n) {
          const int st = n % kStages, round = n / kStages, key = step_at(i) * kKeys;
          for (int ring = 0; ring < n_rings && ok; ++ring) {
            const int slot = ring * kStages + st;
            if (n >= kStages) ok = mbar_wait(bar(Smem::k_empty + slot), (round - 1) & 1, abort_flag);
            if (!ok) break;
            mbar_expect_tx(bar(Smem::k_full + slot), kKvBytes);
            tma_load_5d(smem_base + Smem::k + slot * kKvBytes, &P.map_k, bar(Smem::k_full + slot), 0, at.h, key, row_of(ring), at.b);
          }
          if (HAS_BIAS) {
            for (int ring = 0; ring < (ROWS ? 1 : n_tiles) && ok; ++ring) {
              const int slot = ring * 2 + (n & 1);
              if (n >= 2) ok = mbar_wait(bar(Smem::bias_empty + slot), ((n >> 1) - 1) & 1, abort_flag);
              if (!ok) break;
              mbar_expect_tx(bar(Smem::bias_full + slot), kBiasBytes);
              tma_load_5d(smem_base + Smem::bias + slot * kBiasBytes, &P.map_bias, bar(Smem::bias_full + slot), key, first_query(ring),
                          at.h, P.bias_groups == 1 ? 0 : at.r0, at.b);
            }
          }
          for (int ring = 0; ring < n_rings && ok; ++ring) {
            const int slot = ring * kStages + st;
            if (n >= kStages) ok = mbar_wait(bar(Smem::v_empty + slot), (round - 1) & 1, abort_flag);
            if (!ok) break;
            mbar_expect_tx(bar(Smem::v_full + slot), kKvBytes);
            tma_load_5d(smem_base + Smem::v + slot * kKvBytes, &P.map_v, bar(Smem::v_full + slot), 0, at.h, key, row_of(ring), at.b);
          }
        }
      }
    }
  } else if (warp >= 9 && warp - 9 < n_tiles) {
    // ------------------------------------------------------------------ MMA issuers (one thread per tile)
    const int w = warp - 9, ring = (ROWS ? w : 0) * kStages;
    if (lane == 0 && KS > 0) {
      constexpr uint32_t fmt = Half2<T>::kFormat;
      constexpr uint32_t idesc_qk = instr_desc(fmt, 0, 0, kTile, kKeys);
      constexpr uint32_t idesc_pv = instr_desc(fmt, 0, 1, kTile, kHeadDim);
      const bool signoff = needs_signoff(w);
      const uint32_t s_t = tmem_base + kSCol + w * kKeys, p_t = tmem_base + kPCol + w * (kKeys / 2), o_t = tmem_base + kOCol + w * kHeadDim;
      const uint64_t qdesc = smem_desc(smem_base + Smem::q + w * kQBytes, 16, 512, kSwizzle64B);
      const uint64_t kdesc0 = smem_desc(smem_base + Smem::k + ring * kKvBytes, 16, 512, kSwizzle64B);
      const uint64_t vdesc0 = smem_desc(smem_base + Smem::v + ring * kKvBytes, 16, 512, kSwizzle64B);
      // S[128 x 64] = Q[128 x 32] K[64 x 32]^T; both K-major, 64-byte swizzle: 8-row groups 512 bytes apart,
      // each 16-channel step advances 32 bytes inside the swizzle span.
      auto issue_qk = [&](int st) {
        const uint64_t kdesc = kdesc0 + uint64_t((st * kKvBytes) >> 4);
#pragma unroll
        for (int kk = 0; kk < kHeadDim / 16; ++kk)
          mma_ss(s_t, qdesc + uint64_t(kk * 2), kdesc + uint64_t(kk * 2), idesc_qk, kk > 0 ? 1u : 0u);
        mma_commit(bar(Smem::s_full + w));
        mma_commit(bar(Smem::k_empty + ring + st));
      };
      // O[128 x 32] += P[128 x 64] V[64 x 32]; V is MN-major (channel contiguous), 64-byte swizzle:
      // 8-key groups are 512 bytes apart, each 16-key step advances 1024 bytes.
      auto issue_pv = [&](int st, int i) {
        const uint64_t vdesc = vdesc0 + uint64_t((st * kKvBytes) >> 4);
#pragma unroll
        for (int kk = 0; kk < kKeys / 16; ++kk)
          mma_ts(o_t, p_t + kk * 8, vdesc + uint64_t(kk * (1024 >> 4)), idesc_pv, (i > 0 || kk > 0) ? 1u : 0u);
        mma_commit(bar(Smem::pv_done + w));
        mma_commit(bar(Smem::v_empty + ring + st));
      };
      bool ok = mbar_wait(bar(Smem::q_full + w), 0, abort_flag);
      if (ok) ok = mbar_wait(bar(Smem::k_full + ring), 0, abort_flag);
      if (ok) {
        tc_fence_after_sync();
        issue_qk(0);
        if (PERSIST && KS == 1) mma_commit(bar(Smem::q_empty + w));
      }
      int st = 0, round = 0, n = 0, early = 0;  // steps so far, and those that give their scores back early
      for (int item = int(blockIdx.x), turn = 0; ok && item_there(item, turn); item += int(gridDim.x), ++turn) {
        for (int i = 0; i < KS && ok; ++i, ++n) {
          const int next = st + 1 == kStages ? 0 : st + 1, next_round = next == 0 ? round + 1 : round;
          const bool more = i + 1 < KS, turns = PERSIST && !more && item + int(gridDim.x) < P.items, late = !kEarly || (!PLAIN && i >= full_steps);
          // The next scores (of this item or the next one) overwrite these as soon as the last columns are in registers, or, after a late
          // step, when its probabilities stand.
          auto issue_next = [&]() {
            tc_fence_after_sync();
            issue_qk(next);
            if (PERSIST && (more ? i + 2 == KS : KS == 1)) mma_commit(bar(Smem::q_empty + w));
          };
          if (turns) ok = mbar_wait(bar(Smem::q_full + w), (turn + 1) & 1, abort_flag);
          if (ok && (more || turns)) {
            ok = mbar_wait(bar(Smem::k_full + ring + next), next_round & 1, abort_flag);
            if (!late) {
              if (ok) ok = mbar_wait(bar(Smem::s_free + w), (PLAIN ? n : early) & 1, abort_flag);
              if (!ok) break;
              issue_next();
            }
          }
          if (!PLAIN && !late) ++early;
          if (ok) ok = mbar_wait(bar(Smem::v_full + ring + st), round & 1, abort_flag);
          // a warpgroup signs off the value steps with dropped keys after clearing their rows
          if (ok && signoff && i >= full_steps) {
            const int j = i - full_steps;
            ok = mbar_wait(bar(Smem::v_ready + ring + j % kStages), (j / kStages) & 1, abort_flag);
          }
          if (ok) ok = mbar_wait(bar(Smem::p_full + w), n & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          if (late && (more || turns)) issue_next();
          issue_pv(st, i);
          st = next;
          round = next_round;
        }
      }
    }
  } else if ((warp >> 2) < n_tiles) {
    // ------------------------------------------------------------------ softmax warpgroups
    const int w = warp >> 2, ring = ROWS ? w : 0;
    const int t = tid & (kTile - 1);
    const uint32_t lane_field = uint32_t((warp & 3) * 32) << 16;
    const uint32_t s_tmem = tmem_base + lane_field + kSCol + w * kKeys;
    const uint32_t p_tmem = tmem_base + lane_field + kPCol + w * (kKeys / 2);
    const uint32_t o_tmem = tmem_base + lane_field + kOCol + w * kHeadDim;
    const float c = P.scale * kLog2e;
    const f32x2 c2 = pack2(c, c), log2e2 = pack2(kLog2e, kLog2e);
    const bool signs_off = needs_signoff(w) && (ROWS || w == 0);
    float ref = -INFINITY, l_run = 0.f;  // reference (base-2 logit) and sum of the row
    bool ok = true;
    int base = 0;  // steps of the items before

    // One step; `drops`: some of its keys are dropped.
    auto step = [&](int i, auto drops) {
      constexpr bool kDrops = decltype(drops)::value, kLate = kDrops || !kEarly;
      uint2 bits = make_uint2(0xffffffffu, 0xffffffffu);  // keys 0-31 and 32-63 of the step
      if (kDrops) bits = *reinterpret_cast<const uint2*>(keep_words + ring * kMaxKeepWords + step_at(i) * 2);
      if (kDrops && signs_off) {
        // Values of dropped keys must not reach the tensor core (0 * inf): clear their rows in shared memory.
        const int slot = ring * kStages + i % kStages;
        ok = mbar_wait(bar(Smem::v_full + slot), (i / kStages) & 1, abort_flag);
        if (!ok) return;
        if (t < kKeys && (((t < 32 ? bits.x : bits.y) >> (t & 31)) & 1u) == 0) {
          uint4* row = reinterpret_cast<uint4*>(smem_gen + Smem::v + slot * kKvBytes + t * 64);
          row[0] = row[1] = row[2] = row[3] = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
        mbar_arrive_warp(bar(Smem::v_ready + ring * kStages + (i - full_steps) % kStages));
      }

      const int at_step = base + i;  // over all items: what barrier phases count
      const int bias_slot = (ROWS ? 0 : w * 2) + (at_step & 1);
      // the phases the step needs are probed together: one round trip to the barrier words when all are complete
      const bool s_there = mbar_test(bar(Smem::s_full + w), at_step & 1);
      const bool bias_there = HAS_BIAS && mbar_test(bar(Smem::bias_full + bias_slot), (at_step >> 1) & 1);
      ok = mbar_wait_probed(s_there, bar(Smem::s_full + w), at_step & 1, abort_flag);
      if (ok && HAS_BIAS) ok = mbar_wait_probed(bias_there, bar(Smem::bias_full + bias_slot), (at_step >> 1) & 1, abort_flag);
      if (!ok) return;
      tc_fence_after_sync();
      // swizzled row of the bias tile: 16-byte chunk n holds keys 8 n .. 8 n + 7
      const uint32_t bias_row = smem_base + Smem::bias + bias_slot * kBiasBytes + t * 128 + ((t & 7) << 4);

      // Base-2 logits x + shift of 16 columns, as eight pairs; dropped keys become -inf.
      auto logits16 = [&](int chunk, const uint32_t (&s)[16], const uint4 (&bw)[2], f32x2 shift2, f32x2 (&x)[8]) {
        const uint32_t words[8] = {bw[0].x, bw[0].y, bw[0].z, bw[0].w, bw[1].x, bw[1].y, bw[1].z, bw[1].w};
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          const f32x2 s2 = pack2(__uint_as_float(s[2 * n]), __uint_as_float(s[2 * n + 1]));
          x[n] = fma2(s2, c2, HAS_BIAS ? fma2(Half2<T>::widen(words[n]), log2e2, shift2) : shift2);
          if (kDrops) {
            const uint32_t kept = (chunk < 2 ? bits.x : bits.y) >> ((chunk & 1) * 16 + 2 * n);
            float lo, hi;
            unpack2(x[n], lo, hi);
            if ((kept & 1u) == 0) lo = -INFINITY;
            if ((kept & 2u) == 0) hi = -INFINITY;
            x[n] = pack2(lo, hi);
          }
        }
      };
      // The largest base-2 logit of the step.
      auto step_peak = [&]() -> float {
        float peak = -INFINITY;
#pragma unroll 1
        for (int chunk = 0; chunk < 4; ++chunk) {
          uint32_t s[16];
          uint4 bw[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
          if (HAS_BIAS) {
            bw[0] = lds_v4_at(bias_row ^ uint32_t((chunk * 2) << 4));
            bw[1] = lds_v4_at(bias_row ^ uint32_t((chunk * 2 + 1) << 4));
          }
          tmem_ld16(s_tmem + chunk * 16, s);
          tmem_wait_ld();
          tmem_loaded(s);
          f32x2 x[8];
          logits16(chunk, s, bw, pack2(0.f, 0.f), x);
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            float lo, hi;
            unpack2(x[n], lo, hi);
            peak = max3(peak, lo, hi);
          }
        }
        return peak;
      };
      // Raises the reference of the rows whose step needs it, and rescales what they have summed so far.
      auto raise = [&](bool wanted) -> bool {
        tmem_wait_st();  // probabilities of a pass that is about to be repeated
        const float peak = step_peak();
        const bool raised = wanted && peak > ref;
        const float alpha = raised ? ex2(ref - peak) : 1.f;  // 0 for a row without a reference so far
        if (raised) {
          ref = peak;
          l_run *= alpha;
        }
        if (i > 0 && __any_sync(0xffffffffu, raised)) {
          if (!mbar_wait(bar(Smem::pv_done + w), (at_step - 1) & 1, abort_flag)) return false;
          tc_fence_after_sync();
          uint32_t acc[32];
          tmem_ld32(o_tmem, acc);
          tmem_wait_ld();
          tmem_loaded(acc);
#pragma unroll
          for (int n = 0; n < 32; ++n) acc[n] = __float_as_uint(__uint_as_float(acc[n]) * alpha);
          tmem_st32(o_tmem, acc);
          tmem_wait_st();
        }
        return true;
      };
      // Probabilities of the step into tensor memory; returns their sum.  Before the exponentials of the last columns the
      // scores are given back for the next product, unless the step has to be repeated (`wanted`, only asked where `may_repeat`).
      bool p_free = i == 0;
      bool wanted = ref == -INFINITY, may_repeat = true;
      auto step_pass = [&]() -> float {
        const float shift = ref == -INFINITY ? 0.f : -ref;
        const f32x2 shift2 = pack2(shift, shift);
        f32x2 totals[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
        uint32_t s[2][16], packed[16];
        uint4 bw[2][2] = {{make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)}, {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)}};
        tmem_ld16(s_tmem, s[0]);
        if (HAS_BIAS) {
          bw[0][0] = lds_v4_at(bias_row ^ uint32_t((0) << 4));
          bw[0][1] = lds_v4_at(bias_row ^ uint32_t((1) << 4));
        }
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk) {
          tmem_wait_ld();
          tmem_loaded(s[chunk & 1]);
          if (chunk < 3) {  // the next 16 columns travel under the arithmetic of these
            tmem_ld16(s_tmem + (chunk + 1) * 16, s[(chunk + 1) & 1]);
            if (HAS_BIAS) {
              bw[(chunk + 1) & 1][0] = lds_v4_at(bias_row ^ uint32_t((chunk * 2 + 2) << 4));
              bw[(chunk + 1) & 1][1] = lds_v4_at(bias_row ^ uint32_t((chunk * 2 + 3) << 4));
            }
          }
          f32x2 x[8];
          logits16(chunk, s[chunk & 1], bw[chunk & 1], shift2, x);
          if (chunk == 3 && !kLate) {
            float lo, hi, peak = -INFINITY;
            unpack2(add2(totals[0], totals[1]), lo, hi);
            const float before = lo + hi;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
              unpack2(x[n], lo, hi);
              peak = max3(peak, lo, hi);
            }
            wanted = may_repeat && !(before < kStepSumLimit && peak < kLastColumnsLimit);
            if (__any_sync(0xffffffffu, wanted)) return 0.f;
            tc_fence_before_sync();
            mbar_arrive_warp(bar(Smem::s_free + w));
            if (HAS_BIAS) mbar_arrive_warp(bar(Smem::bias_empty + bias_slot));
          }
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            float lo, hi;
            unpack2(x[n], lo, hi);
            const float p0 = ex2(lo), p1 = ex2(hi);
            totals[n & 1] = add2(totals[n & 1], pack2(p0, p1));
            packed[(chunk & 1) * 8 + n] = Half2<T>::pack(p0, p1);
          }
          if (chunk & 1) {
            if (!p_free) {  // the previous P V product must have finished with the P columns
              ok = mbar_wait(bar(Smem::pv_done + w), (at_step - 1) & 1, abort_flag);
              tc_fence_after_sync();
              p_free = true;
            }
            tmem_st16(p_tmem + (chunk >> 1) * 16, packed);
          }
        }
        float lo, hi;
        unpack2(add2(totals[0], totals[1]), lo, hi);
        return lo + hi;
      };
      float sum = 0.f;
      if (kDrops && !PERSIST && (bits.x | bits.y) == 0u) {
        // The row keeps no key of the step, which is walked for its partner: no look for a reference, no exponentials.  (Without a
        // mask there is no such step.)
        if (!p_free) {
          ok = mbar_wait(bar(Smem::pv_done + w), (at_step - 1) & 1, abort_flag);
          tc_fence_after_sync();
        }
        uint32_t zeros[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) zeros[n] = 0u;
        tmem_st16(p_tmem, zeros);
        tmem_st16(p_tmem + 16, zeros);
      } else {
#pragma unroll 1
        for (int attempt = 0; attempt < 2 && ok; ++attempt) {
          if (__any_sync(0xffffffffu, wanted)) ok = raise(wanted);
          else if (attempt > 0) break;
          if (!ok) return;
          may_repeat = attempt == 0;
          sum = step_pass();
          if (kLate) wanted = !(sum < kStepSumLimit);
        }
      }
      if (!ok) return;
      l_run += sum;
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive_warp(bar(Smem::p_full + w));
      if (kLate && HAS_BIAS) mbar_arrive_warp(bar(Smem::bias_empty + bias_slot));
    };
    for (int item = int(blockIdx.x), turn = 0; ok && item_there(item, turn); item += int(gridDim.x), ++turn, base += KS) {
    if (PERSIST) {
      ref = -INFINITY;
      l_run = 0.f;
    }
    int i = 0;
    for (; i < full_steps && ok; ++i) step(i, std::false_type{});
    if (!PLAIN)
      for (; i < KS && ok; ++i) step(i, std::true_type{});

    if (PERSIST) at = fwd_item<ROWS>(P, item);  // (not held through the steps)
    const int r = row_of(w), h = at.h, b = at.b, q_index = first_query(w) + t;
    const bool stored = q_index < P.cols && (!PERSIST || !ROWS || at.r0 + w < P.rows);
    // Gated epilogue: the thread's 32 gate logits are requested before the wait for the last product, so that their
    // trip from global memory runs under it (the words are not touched until the output row is ready).
    uint4 gate_words[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    if (GATED && P.gate_vec16 && ok && stored) {
      const T* g = reinterpret_cast<const T*>(P.gate) + b * P.g_sb + int64_t(r) * P.g_sr + int64_t(q_index) * P.g_sc + h * P.g_sh;
#pragma unroll
      for (int i = 0; i < 4; ++i) gate_words[i] = ldg_v4_here_if(reinterpret_cast<const uint4*>(g) + i, true);
    }
    if (ok && KS > 0) ok = mbar_wait(bar(Smem::pv_done + w), (base + KS - 1) & 1, abort_flag);
    if (ok) {
      tc_fence_after_sync();
      uint32_t acc[32];
#pragma unroll
      for (int n = 0; n < 32; ++n) acc[n] = 0u;
      if (KS > 0) {  // otherwise no product has written the accumulator
        tmem_ld32(o_tmem, acc);
        tmem_wait_ld();
        tmem_loaded(acc);
      }
      if (stored) {
        if (PLAIN && HAS_BIAS && P.closed && isnan(l_run)) *reinterpret_cast<volatile int*>(smem_gen + Smem::lost_flag) = 1;
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        uint32_t o2[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          o2[i] = Half2<T>::pack(__uint_as_float(acc[2 * i]) * inv, __uint_as_float(acc[2 * i + 1]) * inv);
        auto store_row = [&](void* base, int64_t sb, int64_t sr, int64_t sc, int64_t sh, int vec16, const uint32_t (&w)[16]) {
          T* dst = reinterpret_cast<T*>(base) + b * sb + int64_t(r) * sr + int64_t(q_index) * sc + h * sh;
          if (vec16) {
            uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
            for (int i = 0; i < 4; ++i) d4[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
          } else {
            unsigned short* d0 = reinterpret_cast<unsigned short*>(dst);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              d0[2 * i] = (unsigned short)(w[i] & 0xffffu);
              d0[2 * i + 1] = (unsigned short)(w[i] >> 16);
            }
          }
        };
        if (GATED) {
          // The sigmoid gate of the output projection that follows this operator in a pair block, applied to the
          // 16-bit attention values while they are still in registers: gated = sigmoid(gate) * out.  The ungated
          // values are stored too when the reverse pass will need them.
          if (P.plain) store_row(P.plain, P.p_sb, P.p_sr, P.p_sc, P.p_sh, P.plain_vec16, o2);
          const T* g = reinterpret_cast<const T*>(P.gate) + b * P.g_sb + int64_t(r) * P.g_sr + int64_t(q_index) * P.g_sc + h * P.g_sh;
          uint32_t gw[16];
          if (P.gate_vec16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint4 v = gate_words[i];
              gw[4 * i] = v.x; gw[4 * i + 1] = v.y; gw[4 * i + 2] = v.z; gw[4 * i + 3] = v.w;
            }
          } else {
            const unsigned short* g0 = reinterpret_cast<const unsigned short*>(g);
#pragma unroll
            for (int i = 0; i < 16; ++i) gw[i] = uint32_t(g0[2 * i]) | (uint32_t(g0[2 * i + 1]) << 16);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            // the gate multiplies the attention values as they are returned, i.e. after their 16-bit rounding
            const float s_lo = rcp(1.f + ex2(-Half2<T>::lo(gw[i]) * kLog2e));
            const float s_hi = rcp(1.f + ex2(-Half2<T>::hi(gw[i]) * kLog2e));
            o2[i] = Half2<T>::pack(Half2<T>::lo(o2[i]) * s_lo, Half2<T>::hi(o2[i]) * s_hi);
          }
        }
        store_row(P.out, P.o_sb, P.o_sr, P.o_sc, P.o_sh, P.out_vec16, o2);
        if (P.lse) {
          P.lse[((int64_t(b) * P.rows + r) * P.heads + h) * P.cols + q_index] = l_run > 0.f ? (ref + lg2(l_run)) * kLn2 : 0.f;
        }
      }
    }
    }
  }
}

// A query that holds an infinity has NaN for the zeros of keys that the bias closes.  A row whose kept logits are minus infinity, all of
// them, has no probability all the same: zeros (its log-sum-exp is 0 already).  Asked behind a walk in which a row came out as NaN.
template <typename T, bool GATED, bool ROWS, bool PERSIST>
__device__ __forceinline__ void clear_lost_rows(const FwdParams& P, int tid, int warp) {
  const int w = warp >> 2;
  for (int item = int(blockIdx.x); warp < 8 && item < (PERSIST ? P.items : int(blockIdx.x) + 1); item += int(gridDim.x)) {
    const FwdItem i = fwd_item<ROWS>(P, item);
    const int r = ROWS ? i.r0 + w : i.r0, q = (ROWS ? i.q0 : i.q0 + w * kTile) + (tid & (kTile - 1));
    if (r >= P.rows || q >= P.cols) continue;
    T* out = reinterpret_cast<T*>(P.out) + i.b * P.o_sb + int64_t(r) * P.o_sr + int64_t(q) * P.o_sc + i.h * P.o_sh;
    if (!isnan(float(*out)) || !P.logits.all_minus_infinity<T>(i.b, r, i.h, q, P.cols)) continue;
    const T* gate = reinterpret_cast<const T*>(P.gate) + i.b * P.g_sb + int64_t(r) * P.g_sr + int64_t(q) * P.g_sc + i.h * P.g_sh;
    T* plain = reinterpret_cast<T*>(P.plain) + i.b * P.p_sb + int64_t(r) * P.p_sr + int64_t(q) * P.p_sc + i.h * P.p_sh;
#pragma unroll 1
    for (int c = 0; c < kHeadDim; ++c) {
      out[c] = GATED && isnan(float(gate[c])) ? gate[c] : T(0.f);
      if (GATED && P.plain) plain[c] = T(0.f);
    }
  }
}

template <typename T, bool HAS_BIAS, bool GATED, bool ROWS, bool PERSIST>
__global__ void __launch_bounds__(kFwdThreads, 2) ta_fwd_kernel(const __grid_constant__ FwdParams P) {
  using Smem = FwdSmem<ROWS>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Smem::abort_flag);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + Smem::tmem_slot);
  uint32_t* keep_words = reinterpret_cast<uint32_t*>(smem_gen + Smem::keep);
  volatile int* step_count = reinterpret_cast<volatile int*>(smem_gen + Smem::step_count);
  volatile int* full_count = reinterpret_cast<volatile int*>(smem_gen + Smem::full_count);
  uint16_t* step_list = reinterpret_cast<uint16_t*>(smem_gen + Smem::steps);
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  if (device_failed()) return;

  const FwdItem at = fwd_item<ROWS>(P, int(blockIdx.x));
  const int h = at.h, r0 = at.r0, b = at.b, q0 = at.q0;
  const int n_tiles = PERSIST || (ROWS ? r0 + 1 < P.rows : q0 + kTile < P.cols) ? 2 : 1;
  const int n_rings = ROWS ? n_tiles : 1;
  const bool has_mask = !PERSIST && P.mask != nullptr;
  // Steps need keep-bits when there is a mask or when the last key step is ragged.
  const bool ragged = P.cols % kKeys != 0 && !P.closed;
  const bool has_bits = has_mask || ragged;
  auto row_of = [&](int w) { return ROWS ? (PERSIST ? min(r0 + w, P.rows - 1) : r0 + w) : r0; };

  if (warp == 8) {
    // The producer warp sets the barriers up, a lane each, and requests the queries: both run beside the look at the mask.
    for (int i = lane; i < Smem::num_bars; i += 32) {
      int arrivals = 1;
      if ((i >= Smem::k_empty && i < Smem::v_full) || (i >= Smem::v_empty && i < Smem::v_ready)) arrivals = ROWS ? 1 : n_tiles;
      if (i >= Smem::v_ready && i < Smem::bias_full) arrivals = kTile / 32;
      if (i >= Smem::bias_empty && i < Smem::s_full) arrivals = ROWS ? n_tiles * (kTile / 32) : kTile / 32;
      if (i >= Smem::p_full && i < Smem::pv_done) arrivals = kTile / 32;  // (s_free among them)
      mbar_init(bar(i), arrivals);
    }
    if (lane == 0) {
      *abort_flag = 0;
      *reinterpret_cast<volatile int*>(smem_gen + Smem::lost_flag) = 0;
    }
    fence_barrier_init();
    __syncwarp();
    if (lane == 0) {
      for (int w = 0; w < n_tiles; ++w) {
        mbar_expect_tx(bar(Smem::q_full + w), kQBytes);
        tma_load_5d(smem_base + Smem::q + w * kQBytes, &P.map_q, bar(Smem::q_full + w), 0, h, ROWS ? q0 : q0 + w * kTile, row_of(w), b);
      }
    }
  }
  if (warp == 10 && lane == 0) {
    prefetch_tensormap(&P.map_k);
    prefetch_tensormap(&P.map_v);
    if (HAS_BIAS) prefetch_tensormap(&P.map_bias);
  }
  if (warp == 9) {
    tmem_alloc(smem_base + Smem::tmem_slot, kFwdTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  uint32_t* drop_flags = reinterpret_cast<uint32_t*>(smem_gen + Smem::drop_flags);
  if (has_bits && warp < 8) {
    // one bit per key of the pair row: kept by the mask and inside the row (warps 0-3: first row, 4-7: second row; one
    // row: all warps)
    const int ring = ROWS ? warp >> 2 : 0;
    bool dropped_any = false;
    if (ring < n_rings) {
      const uint8_t* mask_row = has_mask ? P.mask + b * P.m_sb + int64_t(row_of(ring)) * P.m_sr : nullptr;
      // (Two turns of bytes under way: with the pair axes exchanged a lane's byte is a sector of its own, and four take 992 columns, 77 % of the tokens
      // kept, from 1056 to 1084 us; one takes an all-ones mask of 768 from 702 to 720.  Gated: four, 611 columns 409 -> 407, 1000 1543 -> 1532.)
#pragma unroll(GATED ? 4 : 2)
      for (int word = ROWS ? warp & 3 : warp; word < P.k_steps * 2; word += ROWS ? 4 : 8) {
        const int key = word * 32 + lane;
        bool keep = key < P.cols;
        if (keep && has_mask) {
          keep = mask_row[int64_t(key) * P.m_sc] != 0;
          dropped_any |= !keep;
        }
        const uint32_t bits = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) keep_words[ring * kMaxKeepWords + word] = bits;
      }
    }
    dropped_any = __any_sync(0xffffffffu, dropped_any);
    if (lane == 0) drop_flags[warp] = dropped_any ? 1u : 0u;
  }
  __syncthreads();
  bool listed = false;  // the mask drops a key of some row of the CTA
  if (has_mask) {
#pragma unroll
    for (int i = 0; i < 8; ++i) listed |= drop_flags[i] != 0;
  }
  if (listed) {
    // The steps in which every row of the CTA keeps every key, then those in which some row keeps some: padding is neither
    // loaded nor computed.
    if (warp == 0) {
      int full = 0, partial = 0;
      for (int first = 0; first < P.k_steps; first += 32) {
        const int j = first + lane;
        uint32_t any = 0, all = 0xffffffffu;
        if (j < P.k_steps) {
#pragma unroll
          for (int ring = 0; ring < Smem::kv_rings; ++ring) {
            if (ring >= n_rings) break;
            const uint2 words = *reinterpret_cast<const uint2*>(keep_words + ring * kMaxKeepWords + 2 * j);
            any |= words.x | words.y;
            all &= words.x & words.y;
          }
        }
        const bool is_full = any != 0 && all == 0xffffffffu, is_partial = any != 0 && all != 0xffffffffu;
        const uint32_t fulls = __ballot_sync(0xffffffffu, is_full), partials = __ballot_sync(0xffffffffu, is_partial);
        const uint32_t below = (1u << lane) - 1;
        if (is_full) step_list[full + __popc(fulls & below)] = uint16_t(j);
        if (is_partial) step_list[256 + partial + __popc(partials & below)] = uint16_t(j);
        full += __popc(fulls);
        partial += __popc(partials);
      }
      if (lane == 0) {
        *full_count = full;
        *step_count = full + partial;
      }
    }
    __syncthreads();
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Two ends of the kernel, and the question about lost rows behind the walk that asks it: with one end, or the question in the output, what the
  // compiler makes of the listed walk is 1 to 3 % slower.  One end is better for a persistent kernel (300 columns 78.3 -> 77.8 us) and for
  // the gated ones (768 columns 711 -> 705).
  constexpr bool kTwoEnds = !PERSIST && !GATED;
  auto any_lost = [&]() { return HAS_BIAS && P.closed && *reinterpret_cast<volatile int*>(smem_gen + Smem::lost_flag) != 0; };
  if (!listed && !ragged) {
    fwd_walk<T, HAS_BIAS, GATED, ROWS, PERSIST, true>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, at, n_tiles, false);
    if constexpr (kTwoEnds) {
      teardown(abort_flag, tmem_base, 9, kFwdTmemCols);
      if (any_lost()) clear_lost_rows<T, GATED, ROWS, PERSIST>(P, tid, warp);
    }
  } else {
    fwd_walk<T, HAS_BIAS, GATED, ROWS, PERSIST, false>(P, smem_base, smem_gen, abort_flag, tmem_base, tid, warp, lane, at, n_tiles, listed);
    if constexpr (kTwoEnds) teardown(abort_flag, tmem_base, 9, kFwdTmemCols);
  }
  if constexpr (!kTwoEnds) {
    teardown(abort_flag, tmem_base, 9, kFwdTmemCols);
    if (any_lost()) clear_lost_rows<T, GATED, ROWS, PERSIST>(P, tid, warp);
  }
}

// Self-test of the bounded wait: one CTA allocates tensor memory and waits, with a one-millisecond limit, on a barrier
// that nothing ever completes.  The wait gives up, the CTA tears down exactly like a compute kernel whose wait ran
// out (abort flag, grace period, status word, tensor memory freed) and returns by itself.
__global__ void __launch_bounds__(128, 1) wait_limit_selftest_kernel() {
  __shared__ __align__(8) uint64_t barrier_word;
  __shared__ uint32_t tmem_slot_word;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5;
  if (device_failed()) return;
  if (threadIdx.x == 0) {
    abort_word = 0;
    mbar_init(smem_u32(&barrier_word), 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot_word), 32);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_word);
  if (threadIdx.x == 32) mbar_wait(smem_u32(&barrier_word), 0, abort_flag, 1000000ull);
  teardown(abort_flag, tmem_base, 0, 32);
}

}  // namespace

int wait_limit_selftest(cudaStream_t stream) {
  wait_limit_selftest_kernel<<<1, 128, 0, stream>>>();
  count_launch();
  return check_launch("bounded-wait self-test");
}

bool tensor_forward_applies(const oops_ta_problem& p) {
  if (p.dtype != OOPS_TA_BF16 && p.dtype != OOPS_TA_F16) return false;
  if (p.head_dim != kHeadDim) return false;
  if (!pair_ok(p.q, p) || !pair_ok(p.k, p) || !pair_ok(p.v, p)) return false;
  if (p.bias_groups != 0) {
    if (p.bias_dtype != p.dtype || p.bias_sk != 1) return false;
    if ((reinterpret_cast<uintptr_t>(p.bias) & 15) != 0) return false;
    if (!stride_ok(p.bias_sq, p.cols) || !stride_ok(p.bias_sh, p.heads) || !stride_ok(p.bias_sg, p.bias_groups) ||
        !stride_ok(p.bias_sb, p.batch))
      return false;
    if (p.cols == 1) return false;
  }
  if (p.cols > kMaxKeepWords * 32) return false;
  const int64_t ctas = int64_t(p.batch) * p.rows * p.heads * ceil_div(p.cols, kTile);
  return ctas <= 0x7fffffffll;
}

// Rows and columns from which a ragged row's bias is closed: 390 columns 170 -> 162 us with the copy, 500 239 -> 228, 1000 1594 -> 1498; all-ones masks 170 -> 167,
// 238 -> 234, 1578 -> 1541.  A token mask has no use for the copy and pays it (390 columns 145.4 -> 146.8, 700 541 -> 545, 1000 as before), and scattered keys
// (214 -> 216); to look at the mask's first row before the copy is made cost them more (148.1, 217).
constexpr int kClosedCols = 384, kClosedRows = 128, kClosedMaxCols = 4096;
uint64_t tensor_forward_workspace(const oops_ta_problem& p) {
  return bias_closes(p) && p.cols % kKeys != 0 && p.cols >= kClosedCols && p.cols <= kClosedMaxCols && p.rows >= kClosedRows ? closed_bias_bytes(p) : 0;
}

namespace {

bool vec16_ok(const oops_ta_pair& t) {
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 8 == 0 && t.sr % 8 == 0 && t.sc % 8 == 0 && t.sh % 8 == 0;
}

int launch_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, const oops_ta_pair* gate,
                   const oops_ta_pair* plain, cudaStream_t stream) {
  FwdParams P{};
  int status = encode_pair(&P.map_q, p, p.q, kTile, "query");
  if (!status) status = encode_pair(&P.map_k, p, p.k, kKeys, "key");
  if (!status) status = encode_pair(&P.map_v, p, p.v, kKeys, "value");
  if (status) return status;
  const bool has_bias = p.bias_groups != 0;
  const uint64_t scratch = tensor_forward_workspace(p);
  P.closed = scratch != 0 && p.workspace && p.workspace_bytes >= scratch && (reinterpret_cast<uintptr_t>(p.workspace) & 15) == 0;
  if (P.closed) {
    status = close_bias(&P.map_bias, p, p.workspace, "bias", stream);
    if (status) return status;
    P.logits = Logits(p);
  } else if (has_bias) {
    status = encode_bias(&P.map_bias, p, p.bias, p.bias_sq, p.bias_sh, p.bias_sg, p.bias_sb, kTile, "bias");
    if (status) return status;
  }
  P.out = out.ptr;
  P.o_sb = out.sb;
  P.o_sr = out.sr;
  P.o_sc = out.sc;
  P.o_sh = out.sh;
  P.out_vec16 = vec16_ok(out);
  if (gate) {
    P.gate = gate->ptr;
    P.g_sb = gate->sb;
    P.g_sr = gate->sr;
    P.g_sc = gate->sc;
    P.g_sh = gate->sh;
    P.gate_vec16 = vec16_ok(*gate);
    if (plain && plain->ptr) {
      P.plain = plain->ptr;
      P.p_sb = plain->sb;
      P.p_sr = plain->sr;
      P.p_sc = plain->sc;
      P.p_sh = plain->sh;
      P.plain_vec16 = vec16_ok(*plain);
    }
  }
  P.lse = lse;
  P.mask = p.mask;
  P.m_sb = p.mask_sb;
  P.m_sr = p.mask_sr;
  P.m_sc = p.mask_sc;
  P.batch = p.batch;
  P.rows = p.rows;
  P.cols = p.cols;
  P.heads = p.heads;
  P.bias_groups = p.bias_groups;
  // A row-shared bias (or none) pairs rows: one bias tile serves two, and no CTA is half empty at an odd number of
  // query tiles.  A per-row bias has nothing to share between rows; a single row has no partner.
  const bool pair_rows = p.bias_groups <= 1 && p.rows > 1;
  P.q_items = (int)ceil_div(p.cols, pair_rows ? kTile : 2 * kTile);
  P.k_steps = (int)ceil_div(p.cols, kKeys);
  P.scale = p.scale;
  P.items = (int)(int64_t(p.batch) * (pair_rows ? ceil_div(p.rows, 2) : p.rows) * p.heads * P.q_items);
  // Without a mask, a CTA that has a place on an SM goes on to further items as soon as there are more items than places.  It
  // pays where items are short: set-up, first copies and output cost as much as three steps (4 steps, N = 256 and two samples:
  // 76 -> 70 us, 6: 111 -> 107, 8: 240 -> 236 at N = 499; 12: 697 -> 707, the counters of the longer walk cost more).  With a
  // mask every item has a step list of its own, and its CTA to itself.
  const int places = 2 * sm_count();
  const bool persistent = pair_rows && !p.mask && P.k_steps <= 8 && P.items > places;
  const unsigned grid = (unsigned)(persistent ? places : P.items);

  auto launch = [&](auto kernel, int smem) -> int {
    const int rc = reserve_smem(kernel, smem);
    if (rc) return rc;
    kernel<<<grid, kFwdThreads, smem, stream>>>(P);
    count_launch();
    return check_launch("tcgen05 forward");
  };
  auto pick = [&](auto type_tag) -> int {
    using T = decltype(type_tag);
    auto paired = [&](auto rows, auto persist) -> int {
      constexpr bool ROWS = decltype(rows)::value, PERSIST = decltype(persist)::value;
      constexpr int smem = FwdSmem<ROWS>::bytes;
      if (gate)
        return has_bias ? launch(ta_fwd_kernel<T, true, true, ROWS, PERSIST>, smem) : launch(ta_fwd_kernel<T, false, true, ROWS, PERSIST>, smem);
      return has_bias ? launch(ta_fwd_kernel<T, true, false, ROWS, PERSIST>, smem) : launch(ta_fwd_kernel<T, false, false, ROWS, PERSIST>, smem);
    };
    if (persistent) return paired(std::true_type{}, std::true_type{});
    return pair_rows ? paired(std::true_type{}, std::false_type{}) : paired(std::false_type{}, std::false_type{});
  };
  return p.dtype == OOPS_TA_BF16 ? pick(__nv_bfloat16{}) : pick(__half{});
}

}  // namespace

int tensor_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream) {
  return launch_forward(p, out, lse, nullptr, nullptr, stream);
}

int tensor_forward_gated(const oops_ta_problem& p, const oops_ta_pair& gate, const oops_ta_pair& gated,
                         const oops_ta_pair& plain, float* lse, cudaStream_t stream) {
  return launch_forward(p, gated, lse, &gate, &plain, stream);
}

int forward_device_status(int reset) { return read_tu_device_status(reset); }


}  // namespace oops_ta
