// Parameter block of the dense attention and its tensor-core form.
#pragma once
#include "common.cuh"

namespace llmopt {

struct DenseParams {  // lib/metal_parameters.ml:95-117
  uint32_t batches, heads, q_len, k_len, dim, mask_batches, mask_heads, causal;
  float scale;
  uint32_t kv_heads, token_first_output, past_length, token_first_value, mask_dtype;
};
static_assert(sizeof(DenseParams) == 56, "parameter block is 56 bytes");

// csrc/dense_attention_tc.cu; a negative status: not for this kernel, nothing was launched.
int launch_attention_dense_tc(const KernelArgs& args, const DenseParams& p);

}  // namespace llmopt
