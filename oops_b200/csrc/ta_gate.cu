// Sigmoid gate on attention values: gated = sigmoid(gate) * attention, the element-wise core of the reference's
// gate_attention_output (oops/attention/gate/composed.py:47-53, between its two linear maps), and its reverse pass.
// Layout-agnostic: every tensor is a pair tensor (batch, rows, cols, heads, head_dim) with free element strides and a
// contiguous head_dim axis, so the reference's head-major attention layout (*prefix, H, Q, D) and its token-major
// gate layout (*prefix, Q, H*D) are both described by strides (rows = 1, cols = Q).  HBM-bound element-wise work:
// one thread per 8 channels, 16-byte accesses where the addresses allow (2-byte ones took 9 us where 2 do).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "ta_internal.h"

namespace oops_ta {
namespace {

template <typename T>
__device__ __forceinline__ float to_float(T v) { return float(v); }

__device__ __forceinline__ float sigmoid_of(float g) { return 1.f / (1.f + __expf(-g)); }

struct GateShape {
  int batch, rows, cols, heads, head_dim, chunks;  // chunks of 8 channels per (b, r, c, h)
};

__device__ __forceinline__ bool locate(const GateShape& s, int64_t i, int& b, int& r, int& c, int& h, int& d0) {
  const int64_t total = int64_t(s.batch) * s.rows * s.cols * s.heads * s.chunks;
  if (i >= total) return false;
  // a 64-bit division costs more than the rest of the thread; whole columns fit 32 bits on all but giant calls
  const int64_t cells = int64_t(s.heads) * s.chunks;
  uint32_t column, rest;
  if (total <= 0xffffffffll) {
    const uint32_t at = uint32_t(i), per = uint32_t(cells);
    column = at / per;
    rest = at - column * per;
    c = int(column % uint32_t(s.cols));
    column /= uint32_t(s.cols);
    r = int(column % uint32_t(s.rows));
    b = int(column / uint32_t(s.rows));
  } else {
    int64_t wide = i / cells;
    rest = uint32_t(i - wide * cells);
    c = int(wide % s.cols);
    wide /= s.cols;
    r = int(wide % s.rows);
    b = int(wide / s.rows);
  }
  h = int(rest / uint32_t(s.chunks));
  d0 = int(rest % uint32_t(s.chunks)) * 8;
  return true;
}

template <typename T>
__device__ __forceinline__ T* at(const oops_ta_pair& t, int b, int r, int c, int h, int d) {
  return reinterpret_cast<T*>(t.ptr) + b * t.sb + int64_t(r) * t.sr + int64_t(c) * t.sc + int64_t(h) * t.sh + d;
}

// Eight channels; VEC: all of them exist and the address is 16-byte aligned.
template <typename T, bool VEC>
__device__ __forceinline__ void load8(const T* p, int n, float (&v)[8]) {
  if constexpr (VEC) {
    uint4 words[sizeof(T) / 2];
#pragma unroll
    for (int i = 0; i < int(sizeof(T)) / 2; ++i) words[i] = reinterpret_cast<const uint4*>(p)[i];
    const T* e = reinterpret_cast<const T*>(words);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float(e[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < n ? to_float(p[i]) : 0.f;
  }
}
template <typename T, bool VEC>
__device__ __forceinline__ void store8(T* p, int n, const float (&v)[8]) {
  if constexpr (VEC) {
    uint4 words[sizeof(T) / 2];
    T* e = reinterpret_cast<T*>(words);
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = T(v[i]);
#pragma unroll
    for (int i = 0; i < int(sizeof(T)) / 2; ++i) reinterpret_cast<uint4*>(p)[i] = words[i];
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) p[i] = T(v[i]);
  }
}

template <typename T, bool VEC>
__global__ void gate_forward_kernel(GateShape s, oops_ta_pair attention, oops_ta_pair gate, oops_ta_pair out) {
  int b, r, c, h, d0;
  if (!locate(s, int64_t(blockIdx.x) * blockDim.x + threadIdx.x, b, r, c, h, d0)) return;
  const int n = min(8, s.head_dim - d0);
  float a[8], g[8];
  load8<T, VEC>(at<T>(attention, b, r, c, h, d0), n, a);
  load8<T, VEC>(at<T>(gate, b, r, c, h, d0), n, g);
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] *= sigmoid_of(g[i]);
  store8<T, VEC>(at<T>(out, b, r, c, h, d0), n, a);
}

template <typename T, bool VEC>
__global__ void gate_backward_kernel(GateShape s, oops_ta_pair attention, oops_ta_pair gate, oops_ta_pair dout,
                                     oops_ta_pair dattention, oops_ta_pair dgate) {
  int b, r, c, h, d0;
  if (!locate(s, int64_t(blockIdx.x) * blockDim.x + threadIdx.x, b, r, c, h, d0)) return;
  const int n = min(8, s.head_dim - d0);
  float a[8], g[8], up[8];
  load8<T, VEC>(at<T>(attention, b, r, c, h, d0), n, a);
  load8<T, VEC>(at<T>(gate, b, r, c, h, d0), n, g);
  load8<T, VEC>(at<T>(dout, b, r, c, h, d0), n, up);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float sg = sigmoid_of(g[i]);
    a[i] = up[i] * a[i] * sg * (1.f - sg);
    up[i] *= sg;
  }
  if (dattention.ptr) store8<T, VEC>(at<T>(dattention, b, r, c, h, d0), n, up);
  if (dgate.ptr) store8<T, VEC>(at<T>(dgate, b, r, c, h, d0), n, a);
}

// Every 8-channel group of the tensor starts on a 16-byte boundary.
template <typename T>
bool words_ok(const oops_ta_pair& t, int head_dim) {
  const int64_t word = 16 / int64_t(sizeof(T));
  return !t.ptr || (head_dim % 8 == 0 && (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % word == 0 && t.sr % word == 0 &&
                    t.sc % word == 0 && t.sh % word == 0);
}

int check_shape(int dtype, int batch, int rows, int cols, int heads, int head_dim) {
  if (dtype != OOPS_TA_F32 && dtype != OOPS_TA_F16 && dtype != OOPS_TA_BF16)
    return fail(OOPS_TA_UNSUPPORTED_DTYPE, "gate dtype %d is not f32/f16/bf16", dtype);
  if (batch <= 0 || rows <= 0 || cols <= 0 || heads <= 0 || head_dim <= 0)
    return fail(OOPS_TA_INVALID_ARGUMENT, "empty dimension (batch=%d rows=%d cols=%d heads=%d head_dim=%d)", batch, rows, cols,
                heads, head_dim);
  return OOPS_TA_OK;
}

}  // namespace

int gate_forward(int dtype, int batch, int rows, int cols, int heads, int head_dim, const oops_ta_pair& attention,
                 const oops_ta_pair& gate, const oops_ta_pair& out, cudaStream_t stream) {
  int status = check_shape(dtype, batch, rows, cols, heads, head_dim);
  if (status) return status;
  const GateShape s{batch, rows, cols, heads, head_dim, (head_dim + 7) / 8};
  const int64_t total = int64_t(batch) * rows * cols * heads * s.chunks;
  const unsigned grid = (unsigned)ceil_div(total, 256);
  auto launch = [&](auto type) {
    using T = decltype(type);
    const bool vec = words_ok<T>(attention, head_dim) && words_ok<T>(gate, head_dim) && words_ok<T>(out, head_dim);
    (vec ? gate_forward_kernel<T, true> : gate_forward_kernel<T, false>)<<<grid, 256, 0, stream>>>(s, attention, gate, out);
  };
  if (dtype == OOPS_TA_F32) launch(float{});
  else if (dtype == OOPS_TA_F16) launch(__half{});
  else launch(__nv_bfloat16{});
  count_launch();
  return check_launch("gate forward");
}

int gate_backward(int dtype, int batch, int rows, int cols, int heads, int head_dim, const oops_ta_pair& attention,
                  const oops_ta_pair& gate, const oops_ta_pair& dout, const oops_ta_pair& dattention,
                  const oops_ta_pair& dgate, cudaStream_t stream) {
  int status = check_shape(dtype, batch, rows, cols, heads, head_dim);
  if (status) return status;
  const GateShape s{batch, rows, cols, heads, head_dim, (head_dim + 7) / 8};
  const int64_t total = int64_t(batch) * rows * cols * heads * s.chunks;
  const unsigned grid = (unsigned)ceil_div(total, 256);
  auto launch = [&](auto type) {
    using T = decltype(type);
    bool vec = true;
    for (const oops_ta_pair* t : {&attention, &gate, &dout, &dattention, &dgate}) vec = vec && words_ok<T>(*t, head_dim);
    (vec ? gate_backward_kernel<T, true> : gate_backward_kernel<T, false>)<<<grid, 256, 0, stream>>>(s, attention, gate, dout, dattention,
                                                                                                  dgate);
  };
  if (dtype == OOPS_TA_F32) launch(float{});
  else if (dtype == OOPS_TA_F16) launch(__half{});
  else launch(__nv_bfloat16{});
  count_launch();
  return check_launch("gate backward");
}

}  // namespace oops_ta
