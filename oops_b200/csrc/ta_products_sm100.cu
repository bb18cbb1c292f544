// Matrix products of 16-bit operands on tcgen05 with the sigmoid gate of an output projection in their epilogues:
// linear(sigmoid(linear(single, gate_weight)) * attention, output_weight) and its reverse pass (the reference composes them from
// library operations, oops/attention/gate/composed.py:47-53).
//
// A CTA makes one 128 x 64 tile of one product of the launch: a producer warp streams 64-wide slices of both operands through a ring of
// four stages (either operand may lie with its rows or its columns contiguous), one thread issues the products, four warps turn
// the accumulator into the result.  The gate's epilogues read the attention values in their own head-major layout while the product runs.
//
// Token attention's output step is small (2048 rows, 384 and 1024 channels: 1.6 GFLOP a product, 1 us of the tensor pipe), and what it
// costs is launches, on the host above all: two in the forward pass where the library's products and the element-wise gate were
// three, two in the reverse (independent products share a launch) where they were five; 172 -> 92 us of host work a training call.
// On the device a tile waits for its operands from L2 (24 KB per 64 columns at some 45 bytes per clock and SM): 45 us for the call where the
// library's larger tiles and the gate took 39, 18.9 against 19.3 at 64 rows; hence the limit on sizes where the calls are made.
#include <algorithm>
#include <type_traits>

#include "ta_tensor_common.cuh"

namespace oops_ta {
namespace {

using namespace ptx;

constexpr int kBm = 128, kBn = 64, kBk = 64;
constexpr int kStages = 4;
constexpr int kABytes = kBm * kBk * 2, kBBytes = kBn * kBk * 2, kStageBytes = kABytes + kBBytes;
constexpr int kResultWarps = 8, kProducer = 8, kIssuer = 9;
constexpr int kProductThreads = 320;  // two warpgroups of 32 columns each for the result, producer, issuer
constexpr int kProductTmemCols = 64;

struct ProductSmem {
  static constexpr int bars = kStages * kStageBytes;
  static constexpr int full = 0, empty = kStages, done = 2 * kStages, num_bars = done + 1;
  static constexpr int tmem_slot = bars + num_bars * 8;
  static constexpr int abort_flag = tmem_slot + 4;
  static constexpr int failed = abort_flag + 4;
  static constexpr int bytes = failed + 4 + 1024;
};

struct ProductArgs {
  CUtensorMap a, b;
  int first_cta, n_tiles, m, n, k_steps, a_transposed, b_transposed, epilogue;
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
  int count;
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

template <typename T>
__global__ void __launch_bounds__(kProductThreads, 2) ta_products_kernel(const __grid_constant__ ProductsParams P) {
  using Smem = ProductSmem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Smem::abort_flag);
  auto bar = [&](int index) -> uint32_t { return smem_base + Smem::bars + index * 8; };
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int which = 0;
  while (which + 1 < P.count && int(blockIdx.x) >= P.list[which + 1].first_cta) ++which;
  const ProductArgs& A = P.list[which];
  const int tile = int(blockIdx.x) - A.first_cta, m0 = tile / A.n_tiles * kBm, n0 = tile % A.n_tiles * kBn;

  if (warp == kProducer) {
    const bool failed = device_failed();  // (looked at beside the other preparations)
    if (lane < Smem::num_bars) mbar_init(bar(lane), 1);
    fence_barrier_init();
    if (lane == 0) {
      *abort_flag = 0;
      *reinterpret_cast<volatile int*>(smem_gen + Smem::failed) = failed ? 1 : 0;
      prefetch_tensormap(&A.a);
      prefetch_tensormap(&A.b);
    }
  }
  if (warp == kIssuer) {
    tmem_alloc(smem_base + Smem::tmem_slot, kProductTmemCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_gen + Smem::tmem_slot);

  if (*reinterpret_cast<volatile int*>(smem_gen + Smem::failed) != 0) {
    // nothing has been requested: on to the end
  } else if (warp == kProducer) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < A.k_steps && ok; ++i) {
        const int st = i % kStages, k = i * kBk;
        const uint32_t a = smem_base + st * kStageBytes, b = a + kABytes;
        if (i >= kStages) ok = mbar_wait(bar(Smem::empty + st), (i / kStages - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(Smem::full + st), kStageBytes);
        if (A.a_transposed) {
          tma_load_5d(a, &A.a, bar(Smem::full + st), m0, k, 0, 0, 0);
          tma_load_5d(a + kABytes / 2, &A.a, bar(Smem::full + st), m0 + 64, k, 0, 0, 0);
        } else {
          tma_load_5d(a, &A.a, bar(Smem::full + st), k, m0, 0, 0, 0);
        }
        if (A.b_transposed) tma_load_5d(b, &A.b, bar(Smem::full + st), n0, k, 0, 0, 0);
        else tma_load_5d(b, &A.b, bar(Smem::full + st), k, n0, 0, 0, 0);
      }
    }
  } else if (warp == kIssuer) {
    // The whole warp walks the stages (the products' descriptors then stay in uniform registers), and a stage is probed under the products of
    // the one before it: waited for in turn, a stage of four products took 700 clocks, of which the tensor pipe needs 200.
    const uint32_t idesc = instr_desc(Half2<T>::kFormat, A.a_transposed ? 1u : 0u, A.b_transposed ? 1u : 0u, kBm, kBn);
    // columns contiguous (K-major): 8-row groups 1024 bytes apart, 16 columns of k are 32 bytes; rows contiguous: 64-row boxes, 16 rows of k
    // are 2048 bytes
    const uint64_t a_step = (A.a_transposed ? 2048 : 32) >> 4, b_step = (A.b_transposed ? 2048 : 32) >> 4;
    const uint64_t a0 = smem_desc(smem_base, kABytes / 2, 1024, kSwizzle128B), b0 = smem_desc(smem_base + kABytes, 16, 1024, kSwizzle128B);
    bool ok = true, there = false;
    const int k_steps = A.k_steps;
    int st = 0, phase = 0;
    for (int i = 0; i < k_steps && ok; ++i) {
      if (__all_sync(0xffffffffu, there) == 0) ok = mbar_wait_warp(bar(Smem::full + st), phase, abort_flag);
      if (!ok) break;
      const int next = st + 1 == kStages ? 0 : st + 1, next_phase = next == 0 ? phase ^ 1 : phase;
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
  } else {
    const int row = m0 + (tid & (kBm - 1)), first = n0 + (warp >> 2) * 32;
    const bool inside = row < A.m;
    const uint32_t lanes = tmem_base + (uint32_t((warp & 3) * 32) << 16) + (warp >> 2) * 32;
    uint4 values[4], gates[4];
    int64_t value_at = 0, dvalue_at[4] = {0, 0, 0, 0};
    if (A.epilogue != OOPS_TA_PRODUCT_PLAIN) {  // requested ahead of the wait for the product
      const int b = row / A.tokens, q = row - b * A.tokens;
      value_at = b * A.values.sb + int64_t(q) * A.values.sc;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = first + 8 * c, head = n / A.dim, d = n - head * A.dim;
        const bool there = inside && n < A.n;
        values[c] = ldg_v4_here_if(reinterpret_cast<const T*>(A.values.ptr) + value_at + int64_t(head) * A.values.sh + d, there);
        gates[c] = ldg_v4_here_if(reinterpret_cast<const T*>(A.gate) + int64_t(row) * A.gate_ld + n, there && A.epilogue == OOPS_TA_PRODUCT_GATE_REVERSE);
        dvalue_at[c] = b * A.dvalues.sb + int64_t(q) * A.dvalues.sc + int64_t(head) * A.dvalues.sh + d;
      }
    }
    if (mbar_wait(bar(Smem::done), 0, abort_flag)) {
      tc_fence_after_sync();
      uint32_t acc[32];
      tmem_ld32(lanes, acc);
      tmem_wait_ld();
      tmem_loaded(acc);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = first + 8 * c;
        if (!inside || n >= A.n) break;
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(acc[8 * c + e]);
        const uint4 rounded = pack8<T>(x);
        if (A.epilogue != OOPS_TA_PRODUCT_GATE_REVERSE)
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(A.c) + int64_t(row) * A.c_ld + n) = rounded;
        if (A.epilogue == OOPS_TA_PRODUCT_PLAIN) continue;
        float v[8];
        widen8<T>(values[c], v);
        widen8<T>(rounded, x);  // the product as it is stored, or would be
        if (A.epilogue == OOPS_TA_PRODUCT_GATE) {
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
        if (A.gated) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(A.gated) + int64_t(row) * A.gated_ld + n) = pack8<T>(v);
      }
    }
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

}  // namespace

bool products_supported(int dtype, const oops_ta_product* list, int count) {
  if ((dtype != OOPS_TA_BF16 && dtype != OOPS_TA_F16) || count < 1 || count > OOPS_TA_MAX_PRODUCTS) return false;
  int64_t tiles = 0;
  for (int i = 0; i < count; ++i) {
    if (!product_ok(list[i])) return false;
    tiles += tiles_of(list[i]);
  }
  return tiles <= 0x7fffffffll;
}

int products(int dtype, const oops_ta_product* list, int count, cudaStream_t stream) {
  if (!products_supported(dtype, list, count)) return fail(OOPS_TA_UNSUPPORTED_LAYOUT, "products of this type, layout or size are not served");
  ProductsParams P{};
  int64_t grid = 0;
  P.count = count;
  for (int i = 0; i < count; ++i) {
    const oops_ta_product& p = list[i];
    ProductArgs& a = P.list[i];
    int status = encode_operand(&a.a, dtype, p.a, p.a_ld, p.m, p.k, p.a_transposed != 0, kBm, "left operand");
    if (!status) status = encode_operand(&a.b, dtype, p.b, p.b_ld, p.n, p.k, p.b_transposed != 0, kBn, "right operand");
    if (status) return status;
    a.first_cta = (int)grid;
    a.n_tiles = (int)ceil_div(p.n, kBn);
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
    grid += tiles_of(p);
  }
  auto launch = [&](auto kernel) -> int {
    const int status = reserve_smem(kernel, ProductSmem::bytes);
    if (status) return status;
    kernel<<<(unsigned)grid, kProductThreads, ProductSmem::bytes, stream>>>(P);
    count_launch();
    return check_launch("products");
  };
  return dtype == OOPS_TA_BF16 ? launch(ta_products_kernel<__nv_bfloat16>) : launch(ta_products_kernel<__half>);
}

int products_device_status(int reset) { return read_tu_device_status(reset); }

}  // namespace oops_ta
