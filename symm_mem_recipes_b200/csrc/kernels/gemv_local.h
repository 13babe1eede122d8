// Rank-local GEMV (gemv_local.cu) as its callers see it.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include "../device/status.h"

namespace smr {

struct GemvLocalArgs {
  const void* x;          // [batch, K] bf16, batch 1..16, K % 8 == 0, 16-byte aligned
  const void* w;          // [N, K] bf16 when weights_nk, else [K, N]; N % 8 == 0
  void* out;              // [batch, N] bf16 ([batch, N / 2] with silu)
  int batch, K, N;
  bool weights_nk;
  // fused ends (weights_nk only), all optional
  const void* norm_w;     // RMSNorm weight [K]: the product is taken of RMSNorm(x) * norm_w ...
  const float* ss_in;     // ... whose sums of squares are the column sums of ss_in [n_ss][16]
  int n_ss;
  float eps;
  bool silu;              // W = [gate; up], out = SiLU(gate) * up; N % 16 == 0
  const void* residual;   // [batch, N] bf16: out = bf16(bf16(product) + residual)
  float* ss_out;          // [gemv_local_ctas][16]: sums of squares of `out`, one slot per CTA
  // launch: `overlap` = programmatic stream serialization; `static_w` (with it) = the weights were written
  // before the last ordinary launch of this stream, so their stream may start under the predecessor
  bool overlap, static_w;
  int num_sms;
  uint64_t timeout_ns;
  Status* status;
};
int launch_gemv_local(const GemvLocalArgs& args, cudaStream_t stream);
// CTAs of that launch (the slots of ss_out), or a negative cudaError_t.
int gemv_local_ctas(int N, int K, bool weights_nk, bool silu, int num_sms);

}  // namespace smr
