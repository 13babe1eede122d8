// Rank-local GEMV and skinny GEMM (gemv_local.cu) as its callers see it.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include "../device/status.h"

namespace smr {

struct GemvLocalArgs {
  const void* x;          // [batch, K] bf16, batch 1..128 (1..16 with [K, N]), K % 8 == 0, 16-byte aligned
  const void* w;          // [N, K] bf16 when weights_nk, else [K, N]; N % 8 == 0
  void* out;              // [batch, N] bf16 ([batch, N / 2] with a SwiGLU epilogue), 8-byte aligned
  int batch, K, N;
  bool weights_nk;
  int epilogue;           // 0, or SiLU(gate) * up with gate and up rows in groups of 128 (1) or in two halves (2)
  const void* residual;   // [batch, N] bf16 added to the rounded product, or nullptr; epilogue 0
  bool overlap;           // programmatic stream serialization: the set-up may run under the predecessor's end
  int num_sms;
  uint64_t timeout_ns;
  Status* status;
};
int launch_gemv_local(const GemvLocalArgs& args, cudaStream_t stream);

}  // namespace smr
