// Matrix products of 16-bit operands on tcgen05 with the sigmoid gate of an output projection in their epilogues:
// linear(sigmoid(linear(single, gate_weight)) * attention, output_weight) and its reverse pass (the reference composes them from
// library operations, oops/attention/gate/composed.py:47-53).
//
// A CTA makes one 128 x 64 tile of one product of the launch, or a part of its sum: a producer warp streams 64-wide slices of both operands through
// a ring of eight stages (four where two CTAs share an SM; either operand may lie with its rows or its columns contiguous), one warp issues the
// products, eight turn the accumulator into the result.  The gate's epilogues read the attention values in their own head-major layout while the
// product runs.  The parts of a sum are a cluster's CTAs, which add them in their order: results are reproducible.
//
// Token attention's output step is small (2048 rows, 384 and 1024 channels: 1.6 GFLOP a product, 1 us of the tensor pipe), and what it
// costs is launches: two in the forward pass where the library's products and the element-wise gate are three, two in the
// reverse (independent products share a launch) where they are five.  On the device a launch is set-up (1000 clocks, which run under the end of the
// kernel before: programmatic dependent launch), the way of the first operands (900) and a tile's chain of steps.  Times of the whole step
// beside those of the library's products stand where the calls choose (own_products in native.cpp).
#include <algorithm>
#include <type_traits>

#include "ta_tensor_common.cuh"

namespace oops_ta {
namespace {

using namespace ptx;

constexpr int kBm = 128, kBn = 64, kBk = 64;
constexpr int kABytes = kBm * kBk * 2, kBBytes = kBn * kBk * 2, kStageBytes = kABytes + kBBytes;
constexpr int kMostStages = 8, kFewStages = 4;  // a CTA per SM, or two
constexpr int kMostPartBits = 3;                // a sum's parts: the CTAs of a cluster at most
constexpr int kProducer = 8, kIssuer = 9;
constexpr int kProductThreads = 320;  // two warpgroups of 32 columns each for the result, producer, issuer
constexpr int kProductTmemCols = 64;

struct ProductSmem {
  static constexpr int full = 0, empty = kMostStages, done = 2 * kMostStages, num_bars = done + 1;  // in front: barriers and flags
  static constexpr int tmem_slot = num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int stages = 1024;
  static int bytes(int count) { return stages + count * kStageBytes + 1024; }
};
static_assert(ProductSmem::abort_flag + 4 <= ProductSmem::stages, "barriers and flags fit in front of the stages");

struct ProductArgs {
  CUtensorMap a, b;
  int first_cta, tiles, n_tiles, part_bits, m, n, k_steps, a_transposed, b_transposed, epilogue;
  void* c;
  int64_t c_ld;
  oops_ta_pair values, dvalues;
  const void* gate;
  int64_t gate_ld;
  void* gated;
  int64_t gated_ld;
  int tokens, dim;
};
struct ProductsParams {
  ProductArgs list[OOPS_TA_MAX_PRODUCTS];
  int count, stages;
};

// sigmoid(g) and its slope sigmoid(g) * (1 - sigmoid(g)), from e = exp(-|g|) and r = 1 / (1 + e): r or e r, and e r^2.  Nothing cancels where the
// gate is saturated (1 - sigmoid(g) has an error of 2^-25 at best, a tenth of it at g = 14).  1 + e lies in [1, 2], so that the
// approximate reciprocal and one step of Newton's iteration serve as well as a division, which takes the two warpgroups 5 us of a tile.
__device__ __forceinline__ void sigmoid_of(float g, float& s, float& slope) {
  float e;
  asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(-fabsf(g) * kLog2e));  // (subnormal numbers are kept)
  const float d = 1.f + e, r0 = rcp(d), r = fmaf(r0, fmaf(-d, r0, 1.f), r0);
  s = g >= 0.f ? r : e * r;
  slope = e * r * r;
}

template <typename T>
__device__ __forceinline__ void widen8(uint4 words, float (&v)[8]) {
  const uint32_t w[4] = {words.x, words.y, words.z, words.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = Half2<T>::lo(w[i]);
    v[2 * i + 1] = Half2<T>::hi(w[i]);
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(Half2<T>::pack(v[0], v[1]), Half2<T>::pack(v[2], v[3]), Half2<T>::pack(v[4], v[5]), Half2<T>::pack(v[6], v[7]));
}

// The CTAs of a cluster: every thread arrives and waits, and sees what the others wrote to shared memory before.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}
// The next launch may set itself up beside this one; it waits, as this one does, for the end of all before it where it first reads or writes memory.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessors() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void named_barrier_arrive(uint32_t id, uint32_t threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Four f32 at a shared-memory address of this CTA as it lies in CTA `rank` of the cluster.
__device__ __forceinline__ float4 peer_f4(uint32_t address, uint32_t rank) {
  uint32_t there;
  float4 v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(address), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(there) : "memory");
  return v;
}

// Columns 8 c .. 8 c + 7 of a row, for CHUNKS of the chunks c: the sum over 1 << BITS parts in their order, all of whose loads travel together.
template <int BITS, int CHUNKS>
__device__ __forceinline__ void sum_parts(uint32_t from, uint32_t first_rank, uint32_t (&acc)[32]) {
  constexpr int kParts = 1 << BITS;
  float4 v[CHUNKS][kParts][2];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int r = 0; r < kParts; ++r)
#pragma unroll
      for (int j = 0; j < 2; ++j) v[c][r][j] = peer_f4(from + (2 * c + j) * (kBm * 16), first_rank + r);
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float4 sum = v[c][0][j];
#pragma unroll
      for (int r = 1; r < kParts; ++r) sum = make_float4(sum.x + v[c][r][j].x, sum.y + v[c][r][j].y, sum.z + v[c][r][j].z, sum.w + v[c][r][j].w);
      const int at = 8 * c + 4 * j;
      acc[at] = __float_as_uint(sum.x);
      acc[at + 1] = __float_as_uint(sum.y);
      acc[at + 2] = __float_as_uint(sum.z);
      acc[at + 3] = __float_as_uint(sum.w);
    }
}

template <typename T>
__global__ void __launch_bounds__(kProductThreads, 2) ta_products_kernel(const __grid_constant__ ProductsParams P) {
  using Smem = ProductSmem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Smem::abort_flag);
  auto bar = [&](int index) -> uint32_t { return smem_base + index * 8; };
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int which = 0;
  while (which + 1 < P.count && int(blockIdx.x) >= P.list[which + 1].first_cta) ++which;
  const ProductArgs& A = P.list[which];
  const int at = int(blockIdx.x) - A.first_cta, part_bits = A.part_bits, tile = at >> part_bits, part = at & ((1 << part_bits) - 1);
  const int m0 = tile / A.n_tiles * kBm, n0 = tile % A.n_tiles * kBn, stages = P.stages;
  const int step0 = (A.k_steps * part) >> part_bits, k_steps = ((A.k_steps * (part + 1)) >> part_bits) - step0;
  launch_dependents();
  if (tile >= A.tiles) {  // behind the last tile of a cluster's: the others of the cluster meet it at their barriers
    if (part_bits > 0) {
      cluster_sync_all();
      cluster_sync_all();
    }
    return;
  }

  int st = 0, phase = 0, requested = 0;
  auto request = [&]() {
    const int k = (step0 + requested) * kBk;
    const uint32_t a = smem_base + Smem::stages + st * kStageBytes, b = a + kABytes;
    mbar_expect_tx(bar(Smem::full + st), kStageBytes);
    if (A.a_transposed) {
      tma_load_5d(a, &A.a, bar(Smem::full + st), m0, k, 0, 0, 0);
      tma_load_5d(a + kABytes / 2, &A.a, bar(Smem::full + st), m0 + 64, k, 0, 0, 0);
    } else {
      tma_load_5d(a, &A.a, bar(Smem::full + st), k, m0, 0, 0, 0);
    }
    if (A.b_transposed) tma_load_5d(b, &A.b, bar(Smem::full + st), n0, k, 0, 0, 0);
    else tma_load_5d(b, &A.b, bar(Smem::full + st), k, n0, 0, 0, 0);
    ++requested;
    if (++st == stages) {
      st = 0;
      phase ^= 1;
    }
  };
  // The producer warp sets the barriers up and goes on to its requests: nothing that it does waits for the others.
  if (warp == kProducer) {
    if (lane == 0) {
      prefetch_tensormap(&A.a);
      prefetch_tensormap(&A.b);
      *abort_flag = 0;
    }
    if (lane < Smem::num_bars) mbar_init(bar(lane), 1);
    fence_barrier_init();
    __syncwarp();
    named_barrier_arrive(1, kProductThreads);
    wait_for_predecessors();
    if (lane == 0) {
      bool ok = true;
      while (requested < k_steps) {
        if (requested >= stages) ok = mbar_wait(bar(Smem::empty + st), phase ^ 1, abort_flag);
        if (!ok) break;
        request();
      }
    } else if (lane == 1 && device_failed()) {
      *abort_flag = 1;  // a kernel before this one has given up a wait: none of this one's is worth the limit
    }
    __syncwarp();
  } else {
    if (warp == kIssuer) {
      tmem_alloc(smem_base + Smem::tmem_slot, kProductTmemCols);
      tmem_relinquish();
      tc_fence_before_sync();
    }
    named_barrier_sync(1, kProductThreads);
    tc_fence_after_sync();
  }
  // (the producer does not look at it)
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_gen + Smem::tmem_slot);

  // What a result thread makes: chunks of eight columns of its row, four of its warpgroup's 32 columns or, of a sum in parts, its CTA's share.
  const int half = warp >> 2, chunks = part_bits == 3 ? 1 - half : 4 >> part_bits;
  const int chunk0 = part * (8 >> part_bits) + half * chunks, row = m0 + (tid & (kBm - 1)), columns = row < A.m ? min(8 * chunks, A.n - n0 - 8 * chunk0) : 0;
  const uint32_t lanes = tmem_base + (uint32_t((warp & 3) * 32) << 16) + half * 32;
  const int epilogue = A.epilogue;
  uint4 values[4], gates[4];
  int64_t dvalue_at[4] = {0, 0, 0, 0};
  T* const product_row = reinterpret_cast<T*>(A.c) + int64_t(row) * A.c_ld + n0 + 8 * chunk0;
  T* const gated_row = reinterpret_cast<T*>(A.gated) + int64_t(row) * A.gated_ld + n0 + 8 * chunk0;
  uint32_t acc[32];
  bool ok = true;
  if (warp == kIssuer) {
    // The whole warp walks the stages (the products' descriptors then stay in uniform registers), and a stage is probed under the products of
    // the one before it.
    const uint32_t idesc = instr_desc(Half2<T>::kFormat, A.a_transposed ? 1u : 0u, A.b_transposed ? 1u : 0u, kBm, kBn);
    // columns contiguous (K-major): 8-row groups 1024 bytes apart, 16 columns of k are 32 bytes; rows contiguous: 64-row boxes, 16 rows of k
    // are 2048 bytes
    const uint64_t a_step = (A.a_transposed ? 2048 : 32) >> 4, b_step = (A.b_transposed ? 2048 : 32) >> 4;
    const uint64_t a0 = smem_desc(smem_base + Smem::stages, kABytes / 2, 1024, kSwizzle128B);
    const uint64_t b0 = smem_desc(smem_base + Smem::stages + kABytes, 16, 1024, kSwizzle128B);
    bool there = false;
    for (int i = 0; i < k_steps && ok; ++i) {
      if (__all_sync(0xffffffffu, there) == 0) ok = mbar_wait_warp(bar(Smem::full + st), phase, abort_flag);
      if (!ok) break;
      const int next = st + 1 == stages ? 0 : st + 1, next_phase = next == 0 ? phase ^ 1 : phase;
      there = i + 1 < k_steps && mbar_test(bar(Smem::full + next), next_phase);
      tc_fence_after_sync();
      const uint64_t a = a0 + uint64_t((st * kStageBytes) >> 4), b = b0 + uint64_t((st * kStageBytes) >> 4);
#pragma unroll
      for (int kk = 0; kk < kBk / 16; ++kk) mma_ss_warp(tmem_base, a + kk * a_step, b + kk * b_step, idesc, i > 0 || kk > 0 ? 1u : 0u);
      mma_commit_warp(bar(Smem::empty + st));
      st = next;
      phase = next_phase;
    }
    if (ok) mma_commit_warp(bar(Smem::done));
  } else if (warp < kProducer) {
    if (epilogue != OOPS_TA_PRODUCT_PLAIN) {  // requested ahead of the wait for the product
      wait_for_predecessors();
      const int b = row / A.tokens, q = row - b * A.tokens;
      const int64_t value_at = b * A.values.sb + int64_t(q) * A.values.sc;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = n0 + 8 * (chunk0 + c), head = n / A.dim, d = n - head * A.dim;
        const bool take = 8 * c < columns;
        values[c] = ldg_v4_here_if(reinterpret_cast<const T*>(A.values.ptr) + value_at + int64_t(head) * A.values.sh + d, take);
        gates[c] = ldg_v4_here_if(reinterpret_cast<const T*>(A.gate) + int64_t(row) * A.gate_ld + n, take && epilogue == OOPS_TA_PRODUCT_GATE_REVERSE);
        dvalue_at[c] = b * A.dvalues.sb + int64_t(q) * A.dvalues.sc + int64_t(head) * A.dvalues.sh + d;
      }
    }
    ok = mbar_wait(bar(Smem::done), 0, abort_flag);
    if (ok) {
      tc_fence_after_sync();
      tmem_ld32(lanes, acc);
      tmem_wait_ld();
      tmem_loaded(acc);
    }
  }
  // A part of a sum goes to this CTA's shared memory, whose operands every product has read by now: [chunk of eight columns][half][row][four].
  const uint32_t sums = smem_base + Smem::stages + (tid & (kBm - 1)) * 16;
  if (part_bits > 0) {
    if (warp < kProducer && ok) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        sts_v4_at(sums + (half * 8 + j) * (kBm * 16), make_uint4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < kProducer && ok && columns > 0) {
      const uint32_t from = sums + chunk0 * 2 * (kBm * 16), first_rank = cluster_rank() - part;
      if (part_bits == 1) sum_parts<1, 2>(from, first_rank, acc);
      else if (part_bits == 2) sum_parts<2, 1>(from, first_rank, acc);
      else sum_parts<3, 1>(from, first_rank, acc);
    }
  }
  if (warp < kProducer && ok) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (8 * c >= columns) break;
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(acc[8 * c + e]);
      const uint4 rounded = pack8<T>(x);
      if (epilogue != OOPS_TA_PRODUCT_GATE_REVERSE) *reinterpret_cast<uint4*>(product_row + 8 * c) = rounded;
      if (epilogue == OOPS_TA_PRODUCT_PLAIN) continue;
      float v[8];
      widen8<T>(values[c], v);
      widen8<T>(rounded, x);  // the product as it is stored, or would be
      if (epilogue == OOPS_TA_PRODUCT_GATE) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float gate, slope;
          sigmoid_of(x[e], gate, slope);
          v[e] *= gate;
        }
      } else {
        float g[8];
        widen8<T>(gates[c], g);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float gate, slope;
          sigmoid_of(g[e], gate, slope);
          v[e] = x[e] * v[e] * slope;
          x[e] *= gate;
        }
        if (A.dvalues.ptr) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(A.dvalues.ptr) + dvalue_at[c]) = pack8<T>(x);
      }
      if (A.gated) *reinterpret_cast<uint4*>(gated_row + 8 * c) = pack8<T>(v);
    }
  }
  if (part_bits > 0) {
    __syncwarp();
    cluster_sync_all();  // (the others read this CTA's part)
  }
  teardown(abort_flag, tmem_base, kIssuer, kProductTmemCols);
}

// A matrix of `cols` columns whose rows start on 16-byte words; strides of a tensor map are below 2^40 bytes.
bool words(const void* p, int64_t ld, int64_t cols) {
  return p && (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 8 == 0 && ld >= cols && ld < int64_t(1) << 39;
}
bool pair_words(const oops_ta_pair& t) {
  return t.ptr && (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 8 == 0 && t.sc % 8 == 0 && t.sh % 8 == 0;
}

bool product_ok(const oops_ta_product& p) {
  if (p.m <= 0 || p.n <= 0 || p.k <= 0 || p.n % 8 != 0 || p.m > 0x7fffffff - kBm || p.n > 0x7fffffff - kBn || p.k > 0x7fffffff - kBk) return false;
  if (!words(p.a, p.a_ld, p.a_transposed ? p.m : p.k) || !words(p.b, p.b_ld, p.b_transposed ? p.n : p.k)) return false;
  const bool reverse = p.epilogue == OOPS_TA_PRODUCT_GATE_REVERSE;
  if (!reverse && !words(p.c, p.c_ld, p.n)) return false;
  if (p.epilogue == OOPS_TA_PRODUCT_PLAIN) return true;
  if (p.epilogue != OOPS_TA_PRODUCT_GATE && !reverse) return false;
  if (p.tokens <= 0 || p.dim <= 0 || p.dim % 8 != 0 || !pair_words(p.values)) return false;
  if ((p.gated || !reverse) && !words(p.gated, p.gated_ld, p.n)) return false;
  return !reverse || (words(p.gate, p.gate_ld, p.n) && (!p.dvalues.ptr || pair_words(p.dvalues)));
}

int encode_operand(CUtensorMap* map, int dtype, const void* ptr, int64_t ld, int rows, int k, bool transposed, uint32_t box_rows, const char* what) {
  const uint64_t dims[5] = {uint64_t(transposed ? rows : k), uint64_t(transposed ? k : rows), 1, 1, 1};
  const int64_t strides[4] = {ld, 0, 0, 0};
  const uint32_t box[5] = {64, transposed ? uint32_t(kBk) : box_rows, 1, 1, 1};
  return encode_map(map, dtype, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, what);
}

int64_t tiles_of(const oops_ta_product& p) { return ceil_div(p.m, kBm) * ceil_div(p.n, kBn); }

// Parts of a tile's sum, by the steps of 64 that it has.  A CTA walks 430 clocks a step (its copies come in at 57 bytes a clock, alone on its SM or
// not), and the parts meet through their cluster's shared memory in some 1500: sums of more than eight steps are made in up to four
// parts while there is an SM for each CTA, very long ones in eight (in eight throughout, clusters wait for places beside a launch's other product:
// 1024 rows of 8 heads of 32 channels, forward and reverse, 27.4 us and in four 20.4).
int part_bits_of(const oops_ta_product& p) {
  const int64_t steps = ceil_div(p.k, kBk), tiles = tiles_of(p);
  const int most = steps > 128 ? kMostPartBits : 2;
  int bits = 0;
  if (steps > 8)
    while (bits < most && (tiles << (bits + 1)) <= sm_count() && (steps >> (bits + 1)) >= 2) ++bits;
  return bits;
}

}  // namespace

bool products_supported(int dtype, const oops_ta_product* list, int count) {
  if ((dtype != OOPS_TA_BF16 && dtype != OOPS_TA_F16) || count < 1 || count > OOPS_TA_MAX_PRODUCTS) return false;
  int64_t tiles = 0;
  for (int i = 0; i < count; ++i) {
    if (!product_ok(list[i])) return false;
    tiles += (tiles_of(list[i]) + 1) << kMostPartBits;
  }
  return tiles <= 0x7fffffffll;
}

int products(int dtype, const oops_ta_product* list, int count, cudaStream_t stream) {
  if (!products_supported(dtype, list, count)) return fail(OOPS_TA_UNSUPPORTED_LAYOUT, "products of this type, layout or size are not served");
  ProductsParams P{};
  int64_t grid = 0;
  int cluster = 1;
  P.count = count;
  for (int i = 0; i < count; ++i) cluster = std::max(cluster, 1 << part_bits_of(list[i]));
  for (int i = 0; i < count; ++i) {
    const oops_ta_product& p = list[i];
    ProductArgs& a = P.list[i];
    int status = encode_operand(&a.a, dtype, p.a, p.a_ld, p.m, p.k, p.a_transposed != 0, kBm, "left operand");
    if (!status) status = encode_operand(&a.b, dtype, p.b, p.b_ld, p.n, p.k, p.b_transposed != 0, kBn, "right operand");
    if (status) return status;
    a.first_cta = (int)grid;
    a.tiles = (int)tiles_of(p);
    a.n_tiles = (int)ceil_div(p.n, kBn);
    a.part_bits = part_bits_of(p);
    a.m = p.m;
    a.n = p.n;
    a.k_steps = (int)ceil_div(p.k, kBk);
    a.a_transposed = p.a_transposed;
    a.b_transposed = p.b_transposed;
    a.epilogue = p.epilogue;
    a.c = p.c;
    a.c_ld = p.c_ld;
    a.values = p.values;
    a.dvalues = p.dvalues;
    a.gate = p.gate;
    a.gate_ld = p.gate_ld;
    a.gated = p.gated;
    a.gated_ld = p.gated_ld;
    a.tokens = p.tokens;
    a.dim = p.dim;
    grid += ceil_div(tiles_of(p) << a.part_bits, cluster) * cluster;
  }
  // (clusters whose CTAs have an SM each do not find places on all SMs: 36 tiles in four parts, one after the other, 16.1 us and not 10.6)
  P.stages = grid <= (cluster > 1 ? sm_count() * 3 / 4 : sm_count()) ? kMostStages : kFewStages;
  auto launch = [&](auto kernel) -> int {
    const int bytes = ProductSmem::bytes(P.stages), status = reserve_smem(kernel, bytes);
    if (status) return status;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned)grid);
    config.blockDim = dim3(kProductThreads);
    config.dynamicSmemBytes = bytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2]{};
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim = {(unsigned)cluster, 1, 1};
    config.attrs = attributes;
    config.numAttrs = cluster > 1 ? 2 : 1;
    cudaLaunchKernelEx(&config, kernel, P);
    count_launch();
    return check_launch("products");
  };
  return dtype == OOPS_TA_BF16 ? launch(ta_products_kernel<__nv_bfloat16>) : launch(ta_products_kernel<__half>);
}

int products_device_status(int reset) { return read_tu_device_status(reset); }

}  // namespace oops_ta
