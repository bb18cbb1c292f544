// Internal declarations shared by the translation units of liboops_ta_sm100.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "oops_ta.h"

namespace oops_ta {

// Records a message for oops_ta_last_error() and returns `status`.
int fail(int status, const char* format, ...);

// Bumps the process-wide launch counter reported by oops_ta_launch_count().
void count_launch(int n = 1);

// Checks the last launch and converts a CUDA error into a status.
int check_launch(const char* what);

// Allows the kernel `bytes` of dynamic shared memory on the current device; remembered, so that only a kernel's first launch
// on a device asks the driver (1 us a call).
int reserve_dynamic_smem(const void* kernel, int bytes);

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

size_t dtype_size(int dtype);

// Layout-agnostic FFMA kernels (any head_dim <= 256, any strides, f32/f16/bf16).
uint64_t generic_forward_workspace(const oops_ta_problem& p);
uint64_t generic_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g);
int generic_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);
int generic_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                     const oops_ta_grads& g, cudaStream_t stream);

// FFMA kernels that keep the scores on chip (f32, head_dim <= 64, any strides).
bool f32_forward_applies(const oops_ta_problem& p);
bool f32_backward_applies(const oops_ta_problem& p, const oops_ta_grads& g);
uint64_t f32_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g);
int f32_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);
int f32_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                 const oops_ta_grads& g, cudaStream_t stream);

// Register-level matrix-product kernels (f16/bf16, head_dim <= 64, any strides and bias type).
bool mma_applies(const oops_ta_problem& p);
uint64_t mma_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g);
int mma_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);
int mma_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                 const oops_ta_grads& g, cudaStream_t stream);

// tcgen05 kernels of the same calls for bf16 operands without a mask whose rows are 16-byte words.  The reverse is a part of
// mma_backward: row dots, scratch and the sum of the bias gradient's parts are the same.
bool wide_forward_applies(const oops_ta_problem& p, const oops_ta_pair& out);
int wide_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);
bool wide_backward_applies(const oops_ta_problem& p, const oops_ta_pair& dout, const oops_ta_grads& g);
int wide_backward(const oops_ta_problem& p, const oops_ta_pair& dout, const float* lse, const float* delta, const oops_ta_grads& g,
                  int num_parts, float* parts, cudaStream_t stream);
int wide_device_status(int reset);

// Products of 16-bit operands with the gate of an output projection in their epilogues (include/oops_ta.h).
bool products_supported(int dtype, const oops_ta_product* list, int count);
int products(int dtype, const oops_ta_product* list, int count, cudaStream_t stream);
int products_device_status(int reset);

// The layout-agnostic forward pass on the library's built-in scratch array (no caller workspace).
uint64_t static_forward_capacity();
int static_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);

// tcgen05/TMEM/TMA kernels (f16/bf16, head_dim 32, 16-byte aligned rows).
bool tensor_forward_applies(const oops_ta_problem& p);
bool tensor_backward_applies(const oops_ta_problem& p, const oops_ta_grads* g);
uint64_t tensor_forward_workspace(const oops_ta_problem& p);
uint64_t tensor_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g);
int tensor_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream);
int tensor_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse,
                    const oops_ta_grads& g, cudaStream_t stream);

// Sigmoid gate on attention values and its reverse pass (any strides, f32/f16/bf16); a NULL gradient pointer skips it.
int gate_forward(int dtype, int batch, int rows, int cols, int heads, int head_dim, const oops_ta_pair& attention,
                 const oops_ta_pair& gate, const oops_ta_pair& out, cudaStream_t stream);
int gate_backward(int dtype, int batch, int rows, int cols, int heads, int head_dim, const oops_ta_pair& attention,
                  const oops_ta_pair& gate, const oops_ta_pair& dout, const oops_ta_pair& dattention,
                  const oops_ta_pair& dgate, cudaStream_t stream);
// Pair validity of a packed ragged batch (token bytes, samples + 1 cumulative token counts on the device, number of
// 16-cell chunks over all rows); at most packed_pair_mask_max_samples() samples per call.
int packed_pair_mask(const uint8_t* tokens, const int64_t* token_offsets, int samples, int64_t chunks, uint8_t* out,
                     cudaStream_t stream);
int packed_pair_mask_max_samples();
// 16-bit bias of any strides (batch, group, head, query, key) to contiguous rows of ceil(cols / 8) 16-byte words.
int bias_rows(int batch, int groups, int heads, int cols, const void* src, const int64_t strides[5], void* dst, cudaStream_t stream);
// A row-shared bias (rows of whole 16-byte words) in rows of `row` elements (a multiple of 8) that hold `fill` behind the last key.
// With `prefix` (kept keys of every mask row where they are its first ones, else ~0) the launch looks at a sample's rows first.  Where all that
// keep a key keep the same first ones, found[sample] is their number (0: none keeps any) and the bias is closed behind those; else it is ~0.
// Where `whole` (there is nothing to close behind the last key) such a sample is not copied, and none is if no row drops a key: `drops` says
// that of every eight rows of the call.
struct ClosedBiasLook {
  const uint32_t *prefix = nullptr, *drops = nullptr;
  int rows = 0, whole = 0;
  uint32_t* found = nullptr;
};
int closed_bias(int batch, int heads, int cols, const void* src, int64_t s_b, int64_t s_h, int64_t s_q, void* dst, int row, uint16_t fill,
                const ClosedBiasLook& look, cudaStream_t stream);
// Layer normalisation over the last axis of (rows, width) activations (row strides in elements, contiguous rows);
// weight / bias / gradients of them may be NULL; affine_dtype is the activation dtype or f32.
uint64_t layer_norm_backward_workspace_bytes(int64_t rows, int width);
int layer_norm_max_width();
int layer_norm_forward(int dtype, int affine_dtype, int64_t rows, int width, const void* x, int64_t x_stride, const void* weight,
                       const void* bias, float eps, void* y, int64_t y_stride, float* mean, float* rstd, cudaStream_t stream);
int layer_norm_backward(int dtype, int affine_dtype, int64_t rows, int width, const void* dy, int64_t dy_stride, const void* x,
                        int64_t x_stride, const void* weight, const float* mean, const float* rstd, void* dx, int64_t dx_stride,
                        void* dweight, void* dbias, void* workspace, cudaStream_t stream);
// Sums f32 partial rows of the two affine gradients in a fixed order (a NULL tensor is skipped).
int reduce_parameter_parts(int affine_dtype, const float* dw_parts, const float* db_parts, int num_parts, int width, void* dweight,
                           void* dbias, cudaStream_t stream);
// Passes of the triangle multiplicative update between its GEMMs (include/oops_ta.h has the layouts).
int channel_norm_max_width();
int pair_gate_forward(int dtype, int prefix, int tokens, int padded, int hidden, const void* proj, int64_t ld, const void* mask,
                      void* left, void* right, cudaStream_t stream);
int pair_gate_backward(int dtype, int prefix, int tokens, int padded, int hidden, const void* proj, int64_t ld, const void* mask,
                       const void* dleft, const void* dright, void* dproj, int64_t ld_d, cudaStream_t stream);
int channel_norm_forward(int dtype, int affine_dtype, int prefix, int tokens, int padded, int hidden, const void* update,
                         const void* weight, const void* bias, float eps, void* y, float* mean, float* rstd, cudaStream_t stream);
uint64_t channel_norm_backward_workspace_bytes(int dtype, int prefix, int tokens, int padded, int hidden);
int channel_norm_backward(int dtype, int affine_dtype, int prefix, int tokens, int padded, int hidden, const void* dy,
                          const void* update, const void* weight, const float* mean, const float* rstd, void* dupdate,
                          void* dweight, void* dbias, float* workspace, cudaStream_t stream);
int output_gate_forward(int dtype, int64_t rows, int channels, const void* values, const void* gate, int64_t gate_ld, void* out,
                        cudaStream_t stream);
int output_gate_backward(int dtype, int64_t rows, int channels, const void* dout, const void* values, const void* gate,
                         int64_t gate_ld, void* dvalues, void* dgate, int64_t dgate_ld, cudaStream_t stream);
// Forward pass of the tcgen05 kernels with the gate applied in the epilogue: writes sigmoid(gate) * out to `gated`
// and, when plain.ptr is not NULL, the ungated values to `plain`.
int tensor_forward_gated(const oops_ta_problem& p, const oops_ta_pair& gate, const oops_ta_pair& gated,
                         const oops_ta_pair& plain, float* lse, cudaStream_t stream);

// Read (and optionally clear) the device-side status words of the tcgen05 translation units;
// both synchronise with the device.
int forward_device_status(int reset);
// Launches the bounded-wait self-test kernel of the forward translation unit (its wait runs out after 1 ms).
int wait_limit_selftest(cudaStream_t stream);
int backward_device_status(int reset);

}  // namespace oops_ta
