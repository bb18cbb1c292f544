// Bias rows for the TMA kernels: a 16-bit bias (batch, group, head, query, key) of any strides copied to contiguous rows of
// whole 16-byte words, zeros behind the last key.  One launch for what took a permuting copy, a fill and a padding copy.
//
// Bound by latency and, for a bias as a linear map over the pair leaves it (heads innermost), by strided reads.  A thread
// writes one word of eight keys.  Neighbouring threads then take the heads of the same cells where the heads are the
// neighbours in memory, so that a warp's reads share their sectors, and the next words of the row otherwise.
// N = 100, 4 heads: 3.9 -> 2.1 us and one launch less; attention of N = 499 with a projected bias: 260 -> 244 us.
#include "ta_internal.h"

namespace oops_ta {
namespace {

struct BiasRows {
  const uint16_t* src;
  uint16_t* dst;
  int64_t s_b, s_g, s_h, s_q, s_k;
  uint32_t words, heads, cols, groups;  // words of a row
  uint64_t total;
  int heads_inner;
};

// Eight keys of a row from key `word` * 8 on, `fill` (two elements) from key `end` on.  WHOLE: rows of the source are whole 16-byte words.
template <bool WHOLE>
__device__ __forceinline__ uint4 bias_word(const uint16_t* src, int64_t s_k, uint32_t word, uint32_t end, uint32_t fill) {
  uint32_t packed[4] = {fill, fill, fill, fill};
  if (WHOLE && word * 8 + 8 <= end) {
    const uint4 v = *reinterpret_cast<const uint4*>(src + word * 8);
    packed[0] = v.x; packed[1] = v.y; packed[2] = v.z; packed[3] = v.w;
  } else {
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) {
      const uint32_t key = word * 8 + e;
      if (key < end) packed[e / 2] = (packed[e / 2] & (0xffff0000u >> (e % 2 * 16))) | uint32_t(src[int64_t(key) * s_k]) << (e % 2 * 16);
    }
  }
  return make_uint4(packed[0], packed[1], packed[2], packed[3]);
}

// I counts words: 32 bits up to 64 GB of them.  (Whole words of a source that has them are not told apart: the branch costs other biases 3 %, one per row of 300
// columns 126 -> 130 us, and gives those 3 %.)
template <typename I>
__global__ void __launch_bounds__(256) bias_rows_kernel(const BiasRows p) {
  I i = I(blockIdx.x) * 256u + threadIdx.x;
  if (i >= I(p.total)) return;
  uint32_t h = 0, word;
  if (p.heads_inner) {
    h = uint32_t(i % p.heads);
    i /= p.heads;
  }
  word = uint32_t(i % p.words);
  i /= p.words;
  const uint32_t q = uint32_t(i % p.cols);
  i /= p.cols;
  if (!p.heads_inner) {
    h = uint32_t(i % p.heads);
    i /= p.heads;
  }
  const uint32_t g = uint32_t(i % p.groups), b = uint32_t(i / p.groups);
  const uint16_t* src = p.src + b * p.s_b + g * p.s_g + h * p.s_h + q * p.s_q;
  const int64_t row = ((int64_t(b) * p.groups + g) * p.heads + h) * p.cols + q;
  reinterpret_cast<uint4*>(p.dst)[row * p.words + word] = bias_word<false>(src, p.s_k, word, p.cols, 0u);
}

// The bias (batch, head, query, key) in rows of `words` 16-byte words whose keys from an end on are `fill`: the row's end, or a token mask's.
// What no kernel would walk over is not copied.  One launch for all samples; every CTA looks for itself (L2).
struct ClosedBias {
  const uint16_t* src;
  uint16_t* dst;
  int64_t s_b, s_h, s_q;
  uint32_t words, cols, total;  // words of a row, words of a sample
  uint32_t fill;
  ClosedBiasLook look;
};
__global__ void __launch_bounds__(256) closed_bias_kernel(const ClosedBias p) {
  __shared__ uint32_t low[8], high[8];
  const uint32_t b = blockIdx.y;
  uint32_t end = p.cols;
  if (p.look.prefix) {
    uint32_t lo = ~0u, hi = 0u;
    for (int r = threadIdx.x; r < p.look.rows; r += 256) {
      const uint32_t v = p.look.prefix[int64_t(b) * p.look.rows + r];
      if (v != 0) lo = min(lo, v);
      hi = max(hi, v);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
      low[threadIdx.x >> 5] = lo;
      high[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      lo = min(lo, low[i]);
      hi = max(hi, high[i]);
    }
    const bool same = hi == 0 || (lo == hi && hi != ~0u);
    if (blockIdx.x == 0 && threadIdx.x == 0) p.look.found[b] = same ? hi : ~0u;
    if (same && hi != 0) end = hi;
    if (p.look.whole && end == p.cols) {  // closed behind a prefix of another sample, or not walked over
      bool drops = false;
      const uint32_t words = (gridDim.y * uint32_t(p.look.rows) + 7) / 8;
      for (uint32_t i = threadIdx.x; i < words; i += 256) drops |= p.look.drops[i] != 0;
      if (!__syncthreads_or(drops) || !same) return;
    }
  }
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= p.total) return;
  const uint32_t row = i / p.words, word = i - row * p.words, h = row / p.cols, q = row - h * p.cols;
  const uint16_t* src = p.src + b * p.s_b + h * p.s_h + q * p.s_q;
  reinterpret_cast<uint4*>(p.dst)[int64_t(b) * p.total + i] = bias_word<true>(src, 1, word, end, p.fill);
}

}  // namespace

int closed_bias(int batch, int heads, int cols, const void* src, int64_t s_b, int64_t s_h, int64_t s_q, void* dst, int row, uint16_t fill,
                const ClosedBiasLook& look, cudaStream_t stream) {
  const int64_t total = int64_t(heads) * cols * (row / 8);  // of a sample
  if (total == 0 || batch == 0) return OOPS_TA_OK;
  if (total > 0xffffff00ll || batch > 65535) return fail(OOPS_TA_LIMIT_EXCEEDED, "bias of %lld words in %d samples", (long long)total, batch);
  const ClosedBias p{reinterpret_cast<const uint16_t*>(src), reinterpret_cast<uint16_t*>(dst), s_b, s_h, s_q, uint32_t(row / 8), uint32_t(cols),
                     uint32_t(total), fill * 0x10001u, look};
  closed_bias_kernel<<<dim3((unsigned)ceil_div(total, 256), (unsigned)batch), 256, 0, stream>>>(p);
  count_launch();
  return check_launch("closed bias");
}

int bias_rows(int batch, int groups, int heads, int cols, const void* src, const int64_t strides[5], void* dst, cudaStream_t stream) {
  BiasRows p{};
  p.src = reinterpret_cast<const uint16_t*>(src);
  p.dst = reinterpret_cast<uint16_t*>(dst);
  p.s_b = strides[0];
  p.s_g = strides[1];
  p.s_h = strides[2];
  p.s_q = strides[3];
  p.s_k = strides[4];
  p.words = uint32_t(ceil_div(cols, 8));
  p.heads = uint32_t(heads);
  p.cols = uint32_t(cols);
  p.groups = uint32_t(groups);
  p.heads_inner = heads > 1 && p.s_h < p.s_k;
  const int64_t total = int64_t(batch) * groups * heads * cols * p.words;
  if (total == 0) return OOPS_TA_OK;
  if (ceil_div(total, 256) > 0x7fffffffll) return fail(OOPS_TA_LIMIT_EXCEEDED, "bias of %lld words", (long long)total);
  p.total = uint64_t(total);
  const auto kernel = total > 0xffffff00ll ? bias_rows_kernel<uint64_t> : bias_rows_kernel<uint32_t>;
  kernel<<<(unsigned)ceil_div(total, 256), 256, 0, stream>>>(p);
  count_launch();
  return check_launch("bias rows");
}

}  // namespace oops_ta
