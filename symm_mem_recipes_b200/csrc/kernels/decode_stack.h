// One decode step through decoder layers as a single persistent kernel (decode_stack.cu), as its callers see it.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include "../device/status.h"

namespace smr {

struct DecodeStackLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down;   // [N, K] bf16 each; gate_up = [gate; up]
  const void *norm1, *norm2;                      // [H] bf16
  void *k_cache, *v_cache;                        // [batch, s_max, hkv, head_dim] bf16
};

struct DecodeStackArgs {
  const DecodeStackLayer* layers;
  int n_layers;
  const void* x;        // [batch, H] bf16
  void* y;              // [batch, H] bf16
  void* scratch;        // decode_stack_scratch_bytes(...) bytes, contents arbitrary
  size_t scratch_bytes;
  int batch, hidden, ffn, hq, hkv, head_dim, s_max;
  int pos0;
  const int* pos_dev;   // the position, read on the device, or nullptr (then pos0)
  float eps, rope_theta;
  int num_sms;
  uint64_t timeout_ns;
  Status* status;
};
// Whether the kernel takes these shapes on this device (0 = yes, else a cudaError_t).
int decode_stack_supported(int batch, int hidden, int ffn, int hq, int hkv, int head_dim, int s_max, int num_sms);
size_t decode_stack_scratch_bytes(int batch, int hidden, int ffn, int hq, int hkv, int head_dim, int s_max, int num_sms);
int launch_decode_stack(const DecodeStackArgs& args, cudaStream_t stream);

}  // namespace smr
