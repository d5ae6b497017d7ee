// Recurrent-state (gated short convolution) kernels for sm_100a.
// Restatement of lib/metal_recurrent_source.ml:9-269:
//   llmopt_short_conv_f16{,_f32}           depthwise conv1d, channel-major
//   llmopt_short_conv_silu_tm_{f16,f32}    token-major conv + SiLU
//   llmopt_short_conv_step{,_fused}_f16    one decode token, state updated in place
//   llmopt_short_conv_prefill{,_init}_f16  the same recurrence over T tokens
// All arithmetic in fp32, one rounding to half per stored value, as the
// reference kernels do. These move a few KB per call (a prompt some MB); launch
// latency is the bound, so they stay one thread per output element or short strip.
#include "common.cuh"

namespace llmopt {
namespace {

struct ShortConvParams {  // lib/metal_recurrent_source.ml:10-13
  uint32_t batches, channels, input_width, output_width, kernel_width, stride, padding, dilation;
};
struct ShortConvSiluTmParams {  // lib/metal_recurrent_source.ml:67-70
  uint32_t batches, tokens, channels, kernel_width, stride, padding, dilation, output_start;
};

template <typename W>
__global__ void short_conv_kernel(const __half* __restrict__ input, const W* __restrict__ weight,
                                  __half* __restrict__ output, ShortConvParams p) {
  grid_chain_prologue();
  const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= p.batches * p.channels * p.output_width) return;
  const uint32_t position = gid % p.output_width;
  const uint32_t channel = (gid / p.output_width) % p.channels;
  const uint32_t batch = gid / (p.output_width * p.channels);
  float accumulator = 0.0f;
  for (uint32_t tap = 0; tap < p.kernel_width; ++tap) {
    const int source = (int)(position * p.stride) - (int)p.padding + (int)(tap * p.dilation);
    if (source >= 0 && source < (int)p.input_width)
      accumulator += __half2float(input[((size_t)batch * p.channels + channel) * p.input_width + (uint32_t)source]) *
                     (float)weight[channel * p.kernel_width + tap];
  }
  output[gid] = __float2half_rn(accumulator);
}

template <typename W>
__global__ void short_conv_silu_tm_kernel(const __half* __restrict__ input, const W* __restrict__ weight,
                                          __half* __restrict__ output, ShortConvSiluTmParams p) {
  grid_chain_prologue();
  const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= p.batches * p.tokens * p.channels) return;
  const uint32_t channel = gid % p.channels;
  const uint32_t token = (gid / p.channels) % p.tokens;
  const uint32_t batch = gid / (p.tokens * p.channels);
  float accumulator = 0.0f;
  for (uint32_t tap = 0; tap < p.kernel_width; ++tap) {
    const int source = (int)((token + p.output_start) * p.stride) - (int)p.padding + (int)(tap * p.dilation);
    if (source >= 0 && source < (int)p.tokens)
      accumulator += __half2float(input[((size_t)batch * p.tokens + (uint32_t)source) * p.channels + channel]) *
                     (float)weight[channel * p.kernel_width + tap];
  }
  // the convolved value is rounded to half before SiLU (lib/metal_recurrent_source.ml:94-96)
  const float value = __half2float(__float2half_rn(accumulator));
  output[gid] = __float2half_rn(value / (1.0f + expf(-value)));
}

// One decode token of gridDim.y sequences, whose rows, states and outputs lie `stride` bytes apart (the weights are shared).
__global__ void short_conv_step_kernel(const __half* __restrict__ in_proj, __half* __restrict__ conv_state,
                                       const __half* __restrict__ conv_weight, __half* __restrict__ output,
                                       uint32_t channels, ShortConvStepStrides stride) {
  grid_chain_prologue();
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  in_proj = (const __half*)((const uint8_t*)in_proj + blockIdx.y * stride.in_proj);
  conv_state = (__half*)((uint8_t*)conv_state + blockIdx.y * stride.state);
  output = (__half*)((uint8_t*)output + blockIdx.y * stride.output);
  const float x0 = __half2float(in_proj[c]);
  const float x1 = __half2float(in_proj[channels + c]);
  const float x2 = __half2float(in_proj[2 * channels + c]);
  const float g = x0 * x2;
  const float s0 = __half2float(conv_state[c * 3 + 1]);
  const float s1 = __half2float(conv_state[c * 3 + 2]);
  const float s2 = g;
  conv_state[c * 3 + 0] = __float2half_rn(s0);
  conv_state[c * 3 + 1] = __float2half_rn(s1);
  conv_state[c * 3 + 2] = __float2half_rn(s2);
  const float w0 = __half2float(conv_weight[c * 3 + 0]);
  const float w1 = __half2float(conv_weight[c * 3 + 1]);
  const float w2 = __half2float(conv_weight[c * 3 + 2]);
  const float conv_out = s0 * w0 + s1 * w1 + s2 * w2;
  output[c] = __float2half_rn(x1 * conv_out);
}

// A prompt.  An output reads the gated inputs x0 x2 of its own and the two tokens before it and nothing that another
// token's output leaves behind, so a thread takes a strip of `strip` tokens of one channel and forms the two products ahead
// of its strip again: 333 tokens of 1024 channels as one strip per channel (four thread blocks that walk over the prompt,
// every load waiting for the one before) took 101 us, in strips of eight 3 us.  Eight tokens re-read a quarter more rows,
// which still are in the cache; shorter strips would re-read more and 148 SMs are filled already.
constexpr uint32_t kConvStrip = 8;

__global__ void short_conv_prefill_kernel(const __half* __restrict__ in_proj, const __half* __restrict__ conv_weight,
                                          __half* __restrict__ output, __half* state_out, const __half* state_in,
                                          uint32_t tokens, uint32_t channels, uint32_t strip) {
  grid_chain_prologue();
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  const uint32_t first = blockIdx.y * strip;
  const uint32_t last = min(tokens, first + strip);
  const float w0 = __half2float(conv_weight[c * 3 + 0]);
  const float w1 = __half2float(conv_weight[c * 3 + 1]);
  const float w2 = __half2float(conv_weight[c * 3 + 2]);
  // the gated input `back` places ahead of the strip; ahead of the prompt it is the initial state
  auto before = [&](uint32_t back) {
    if (first >= back) {
      const __half* row = in_proj + (size_t)(first - back) * 3 * channels + c;
      return __half2float(row[0]) * __half2float(row[2 * channels]);
    }
    return state_in != nullptr ? __half2float(state_in[c * 3 + 3 + first - back]) : 0.0f;
  };
  float prev3 = before(3), prev2 = before(2), prev1 = before(1);
#pragma unroll 8
  for (uint32_t t = first; t < last; ++t) {
    const size_t offset = (size_t)t * 3 * channels + c;
    const float x0 = __half2float(in_proj[offset]);
    const float x1 = __half2float(in_proj[offset + channels]);
    const float x2 = __half2float(in_proj[offset + 2 * channels]);
    const float current = x0 * x2;
    const float conv_out = prev2 * w0 + prev1 * w1 + current * w2;
    output[(size_t)t * channels + c] = __float2half_rn(x1 * conv_out);
    prev3 = prev2;
    prev2 = prev1;
    prev1 = current;
  }
  if (last == tokens) {
    state_out[c * 3 + 0] = __float2half_rn(prev3);
    state_out[c * 3 + 1] = __float2half_rn(prev2);
    state_out[c * 3 + 2] = __float2half_rn(prev1);
  }
}

}  // namespace

// Buffers [input, weight, output]; params 32 bytes (lib/metal_dispatch_recurrent.ml:175-180).
template <bool WEIGHT_F32>
int launch_short_conv(const KernelArgs& args) {
  ShortConvParams p;
  LLMOPT_REQUIRE(args.buffer_count == 3 && args.param_bytes == sizeof(p), "expects 3 buffers and 32 parameter bytes");
  memcpy(&p, args.params, sizeof(p));
  const size_t count = (size_t)p.batches * p.channels * p.output_width;
  LLMOPT_REQUIRE(args.lengths[0] >= (size_t)p.batches * p.channels * p.input_width * 2, "input buffer is too short");
  LLMOPT_REQUIRE(args.lengths[1] >= (size_t)p.channels * p.kernel_width * (WEIGHT_F32 ? 4 : 2), "weight buffer is too short");
  LLMOPT_REQUIRE(args.lengths[2] >= count * 2, "output buffer is too short");
  if (count == 0) return 0;
  const uint32_t blocks = (uint32_t)((count + 255) / 256);
  if (WEIGHT_F32)
    launch_kernel(args, short_conv_kernel<float>, dim3(blocks), dim3(256), 0, (const __half*)args.buffers[0], (const float*)args.buffers[1],
                                                              (__half*)args.buffers[2], p);
  else
    launch_kernel(args, short_conv_kernel<__half>, dim3(blocks), dim3(256), 0, (const __half*)args.buffers[0], (const __half*)args.buffers[1],
                                                               (__half*)args.buffers[2], p);
  return check_launch(args);
}
template int launch_short_conv<false>(const KernelArgs&);
template int launch_short_conv<true>(const KernelArgs&);

// Buffers [input, weight, output]; params 32 bytes (lib/metal_dispatch_recurrent.ml:210-217).
template <bool WEIGHT_F32>
int launch_short_conv_silu_tm(const KernelArgs& args) {
  ShortConvSiluTmParams p;
  LLMOPT_REQUIRE(args.buffer_count == 3 && args.param_bytes == sizeof(p), "expects 3 buffers and 32 parameter bytes");
  memcpy(&p, args.params, sizeof(p));
  const size_t count = (size_t)p.batches * p.tokens * p.channels;
  LLMOPT_REQUIRE(args.lengths[0] >= count * 2 && args.lengths[2] >= count * 2, "input or output buffer is too short");
  LLMOPT_REQUIRE(args.lengths[1] >= (size_t)p.channels * p.kernel_width * (WEIGHT_F32 ? 4 : 2), "weight buffer is too short");
  if (count == 0) return 0;
  const uint32_t blocks = (uint32_t)((count + 255) / 256);
  if (WEIGHT_F32)
    launch_kernel(args, short_conv_silu_tm_kernel<float>, dim3(blocks), dim3(256), 0,
        (const __half*)args.buffers[0], (const float*)args.buffers[1], (__half*)args.buffers[2], p);
  else
    launch_kernel(args, short_conv_silu_tm_kernel<__half>, dim3(blocks), dim3(256), 0,
        (const __half*)args.buffers[0], (const __half*)args.buffers[1], (__half*)args.buffers[2], p);
  return check_launch(args);
}
template int launch_short_conv_silu_tm<false>(const KernelArgs&);
template int launch_short_conv_silu_tm<true>(const KernelArgs&);

// Buffers [in_proj [3C], conv_state [C,3] (in/out), conv_weight [C,3], output [C]];
// params {channels} (lib/metal_dispatch_recurrent.ml:91-113).
int launch_short_conv_step(const KernelArgs& args) {
  LLMOPT_REQUIRE(args.buffer_count == 4 && args.param_bytes == 4, "expects 4 buffers and 4 parameter bytes");
  const uint32_t channels = param_u32(args, 0);
  LLMOPT_REQUIRE(channels > 0, "needs channels > 0");
  LLMOPT_REQUIRE(args.lengths[0] >= (size_t)channels * 6 && args.lengths[1] >= (size_t)channels * 6 &&
                     args.lengths[2] >= (size_t)channels * 6 && args.lengths[3] >= (size_t)channels * 2,
                 "buffer is too short");
  launch_kernel(args, short_conv_step_kernel, dim3((channels + 255) / 256, 1), dim3(256), 0,
      (const __half*)args.buffers[0], (__half*)args.buffers[1], (const __half*)args.buffers[2], (__half*)args.buffers[3],
      channels, ShortConvStepStrides{});
  return check_launch(args);
}

// The same record of `count` sequences, one after another in a dispatch list, as one launch.  `args` are the first one's,
// `second` the buffers of the second; every further one has to lie as far behind its predecessor (the caller has compared
// them).  False where the records could touch each other's data, which a launch would then read or write in another order.
bool short_conv_steps_stride(const KernelArgs& first, const KernelArgs& second, uint32_t count, ShortConvStepStrides* stride) {
  if (first.buffer_count != 4 || first.param_bytes != 4 || count > 65535) return false;
  const size_t channels = param_u32(first, 0);
  const size_t bytes[4] = {channels * 6, channels * 6, channels * 6, channels * 2};  // of a record in each buffer
  size_t step[4], extent[4];
  for (int i = 0; i < 4; ++i) {
    const intptr_t distance = (const uint8_t*)second.buffers[i] - (const uint8_t*)first.buffers[i];
    if (first.lengths[i] < bytes[i] || distance < 0 || (i == 2 ? distance != 0 : distance < (intptr_t)bytes[i])) return false;
    step[i] = (size_t)distance;
    extent[i] = step[i] * (count - 1) + bytes[i];
  }
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < i; ++j) {
      const uint8_t *a = (const uint8_t*)first.buffers[i], *b = (const uint8_t*)first.buffers[j];
      if (a < b + extent[j] && b < a + extent[i]) return false;
    }
  *stride = ShortConvStepStrides{step[0], step[1], step[3]};
  return true;
}

// Sixteen sequences of 1024 channels: sixteen launches of 1.3 us behind each other in a plan, together one of 2 us.
int launch_short_conv_steps(const KernelArgs& args, uint32_t count, const ShortConvStepStrides& stride) {
  const uint32_t channels = param_u32(args, 0);
  LLMOPT_REQUIRE(channels > 0, "needs channels > 0");
  launch_kernel(args, short_conv_step_kernel, dim3((channels + 255) / 256, count), dim3(256), 0,
      (const __half*)args.buffers[0], (__half*)args.buffers[1], (const __half*)args.buffers[2], (__half*)args.buffers[3],
      channels, stride);
  return check_launch(args);
}

// llmopt_short_conv_prefill_f16: buffers [in_proj, conv_weight, output, state_out
// (, state_in after the parameter slot)]; the _init form binds state_in as the
// fifth buffer (lib/metal_recurrent_source.ml:254-269). params {tokens, channels,
// has_initial_state}.
int launch_short_conv_prefill(const KernelArgs& args) {
  LLMOPT_REQUIRE((args.buffer_count == 4 || args.buffer_count == 5) && args.param_bytes == 12,
                 "expects 4 or 5 buffers and 12 parameter bytes");
  const uint32_t tokens = param_u32(args, 0), channels = param_u32(args, 1), has_initial = param_u32(args, 2);
  LLMOPT_REQUIRE(channels > 0, "needs channels > 0");
  LLMOPT_REQUIRE(args.lengths[0] >= (size_t)tokens * channels * 6 && args.lengths[1] >= (size_t)channels * 6 &&
                     args.lengths[2] >= (size_t)tokens * channels * 2 && args.lengths[3] >= (size_t)channels * 6,
                 "buffer is too short");
  const __half* state_in = nullptr;
  if (args.buffer_count == 5) {
    LLMOPT_REQUIRE(args.lengths[4] >= (size_t)channels * 6, "initial state buffer is too short");
    state_in = (const __half*)args.buffers[4];
  }
  if (has_initial == 0) state_in = nullptr;
  // One strip, whose thread reads ahead of what it writes, where strips would write what others still read: a state
  // updated in place (read by the first strip, written by the last one), outputs or the state in the memory of the projected
  // rows (a token's output can take the place of an input of its own channel that is read by then).  So too for prompts whose
  // strips are more than a grid has rows.
  const size_t state_bytes = (size_t)channels * 6;
  auto overlap = [](const void* a, size_t a_bytes, const void* b, size_t b_bytes) {
    return (uintptr_t)a < (uintptr_t)b + b_bytes && (uintptr_t)b < (uintptr_t)a + a_bytes;
  };
  bool in_place = false;
  for (int written = 2; written < 4; ++written) {
    const void* target = args.buffers[written];
    const size_t bytes = written == 2 ? (size_t)tokens * channels * 2 : state_bytes;
    in_place = in_place || overlap(target, bytes, args.buffers[0], (size_t)tokens * channels * 6) ||
               (state_in != nullptr && overlap(target, bytes, state_in, state_bytes));
  }
  const uint32_t strips = in_place || tokens == 0 ? 1 : (tokens + kConvStrip - 1) / kConvStrip;
  const uint32_t strip = strips == 1 || strips > 65535 ? tokens : kConvStrip;
  launch_kernel(args, short_conv_prefill_kernel, dim3((channels + 255) / 256, strips > 65535 ? 1 : strips), dim3(256), 0,
      (const __half*)args.buffers[0], (const __half*)args.buffers[1], (__half*)args.buffers[2], (__half*)args.buffers[3],
      state_in, tokens, channels, strip);
  return check_launch(args);
}

}  // namespace llmopt
