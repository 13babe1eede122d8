// Attention of one decode step (one new token per sequence) for this rank's heads, split along the cached
// sequence ("flash decoding").  No upstream counterpart (the upstream recipes stop at the single fused op).
//
//     out[b, h, :] = softmax(q[b, h] . K[b, 0..pos, h / G] / sqrt(D)) V[b, 0..pos, h / G]      G = hq / hkv
//
// What bounds it: the cache crosses HBM once (2 * D * 2 bytes per position and KV head); with a short
// context, the chain of dependent steps from the launch to the merged result.
//   * The products are decode_attention.cuh's: mma.sync straight from global memory fragments.  Sixteen warps an
//     SM (two CTAs) keep 64-128 KB in flight.
//   * The warps of a CTA merge through shared memory, the CTAs of a (sequence, KV head) through scratch
//     memory: the last one to arrive adds the others up.
// The new token's key and value come from the QKV row (its warp also writes them into the caches), so no CTA
// depends on another's cache write.  The position may come from device memory and the grid does not depend
// on it: a captured graph serves every position.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../device/vec.cuh"
#include "decode_attention.cuh"
#include "launch.h"
#include "residency.h"

namespace smr {

namespace {

constexpr int kWarps = 8;
constexpr int kMaxSplit = 64;           // CTAs per (sequence, KV head) at most
using attn::kHeads;
using attn::kNoScore;
using attn::kTile;

template <int D>
__global__ void __launch_bounds__(kWarps * 32, 2)
decode_attention_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache,
                        __nv_bfloat16* __restrict__ out, float* scratch, unsigned int* counters, int hq, int hkv,
                        int s_max, int pos0, const int* __restrict__ pos_dev, float scale, float log2_theta) {
  constexpr int kRow = D + 2;                                  // D weighted-V sums, then max and sum
  constexpr int NI = D / 64;                                   // 16-byte loads of a V row
  __shared__ float sm[kWarps][kHeads][kRow];
  __shared__ float split_w[kHeads][kMaxSplit];                 // the last CTA's weights of the splits, per head
  __shared__ float head_sum[kHeads];
  __shared__ __align__(16) float2 angles[D / 2];               // (cos, sin) of the new token's position
  __shared__ int is_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int bh = blockIdx.x, b = bh / hkv, kvh = bh - b * hkv;
  const int n_split = gridDim.y, split = blockIdx.y;
  const int n_units = n_split * kWarps, unit = warp * n_split + split;
  const int G = hq / hkv;
  int pos = pos_dev != nullptr ? *pos_dev : pos0;
  pos = pos < 0 ? 0 : (pos >= s_max ? s_max - 1 : pos);
  const size_t pitch = (size_t)hkv * D;                        // elements between positions
  __nv_bfloat16* kc = k_cache + ((size_t)b * s_max * hkv + kvh) * D;
  __nv_bfloat16* vc = v_cache + ((size_t)b * s_max * hkv + kvh) * D;

  if (log2_theta != 0.f) {
    attn::fill_angles<D>(angles, threadIdx.x, pos, log2_theta);
    __syncthreads();
  }
  const __nv_bfloat16* row = qkv + (size_t)b * (hq + 2 * hkv) * D;
  attn::State<D> st;
  attn::attend<D, false>(kc, vc, pitch, pos, unit, n_units, G, scale, log2_theta != 0.f ? angles : nullptr, [] {},
                  [&](int part, int head, int d) {
                    const int h = part == 0 ? kvh * G + head : (part == 1 ? hq + kvh : hq + hkv + kvh);
                    return ld_16(row + (size_t)h * D + d);
                  },
                  st);
  const float m_run = st.m, l_run = st.l;
  auto& acc = st.acc;

  // ---- the CTA's warps merge through shared memory into one partial per CTA ----
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
      for (int e = 0; e < 4; ++e) sm[warp][2 * t + (e & 1)][i * 64 + g * 8 + 2 * w + (e >> 1)] = acc[i * 4 + w][e];
  if (t == 0) {
    sm[warp][g][D] = m_run;
    sm[warp][g][D + 1] = l_run;
  }
  __syncthreads();
  constexpr int kItems = kHeads * D / (kWarps * 32);           // (head, dimension) items per thread at most
  float* mine = scratch + ((size_t)bh * n_split + split) * kHeads * kRow;
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int item = threadIdx.x + it * kWarps * 32;
    const int h = item / D, d = item % D;
    if (h < G) {
      float big = kNoScore;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) big = fmaxf(big, sm[w][h][D]);
      float sum = 0.f, a = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float f = exp2f(sm[w][h][D] - big);              // 0 for a warp that saw no position while another did
        sum += f * sm[w][h][D + 1];
        a += f * sm[w][h][d];
      }
      if (n_split == 1) {
        out[((size_t)b * hq + kvh * G + h) * D + d] = __float2bfloat16_rn(a / sum);
      } else {
        mine[h * kRow + d] = a;
        if (d == 0) {
          mine[h * kRow + D] = big;
          mine[h * kRow + D + 1] = sum;
        }
      }
    }
  }
  if (n_split == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&counters[bh], 1u) == (unsigned int)(n_split - 1);
  __syncthreads();
  if (!is_last) return;
  // ---- the last CTA of this (b, kv head) merges the CTAs' partials ----
  // Warp h first turns head h's maxima and sums of the splits into one weight per split (a lane takes up to
  // two splits) and the head's total; then every thread adds up its (head, dimension) items over the
  // splits with those weights, eight splits' loads in flight for each of its items.
  __threadfence();
  static_assert(kWarps >= kHeads && kMaxSplit <= 64, "a warp per head, two splits per lane");
  const float* all = scratch + (size_t)bh * n_split * kHeads * kRow;
  if (warp < G) {
    float mv[2], lv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u;
      const float* rec = all + ((size_t)i * kHeads + warp) * kRow + D;
      mv[u] = i < n_split ? __ldcg(rec) : kNoScore;
      lv[u] = i < n_split ? __ldcg(rec + 1) : 0.f;
    }
    float big = fmaxf(mv[0], mv[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    float total = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u;
      const float w = i < n_split ? exp2f(mv[u] - big) : 0.f;  // 0 for a split that saw no position while another did
      split_w[warp][i] = w;
      total += w * lv[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) head_sum[warp] = total;
  }
  __syncthreads();
  float tot[kItems];
#pragma unroll
  for (int it = 0; it < kItems; ++it) tot[it] = 0.f;
#pragma unroll 8
  for (int i = 0; i < n_split; ++i) {
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const int item = threadIdx.x + it * kWarps * 32;
      const int h = item / D, d = item % D;
      if (h < G) tot[it] += split_w[h][i] * __ldcg(all + ((size_t)i * kHeads + h) * kRow + d);
    }
  }
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int item = threadIdx.x + it * kWarps * 32;
    const int h = item / D, d = item % D;
    if (h < G) out[((size_t)b * hq + kvh * G + h) * D + d] = __float2bfloat16_rn(tot[it] / head_sum[h]);
  }
  if (threadIdx.x == 0) counters[bh] = 0u;            // ready for the next launch
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Two CTAs per SM over all (sequence, KV head): rounded down, so that no CTA is left for a second wave that
// would double the time.  A CTA's eight warps take 16 positions each, so more splits than s_max / 128 would
// leave CTAs without a tile even at the end of the context; few enough for one CTA to combine them.
int splits_for(int rows, int s_max) {
  int n = 2 * device_sms() / (rows > 0 ? rows : 1);
  const int by_length = (s_max + kTile * kWarps - 1) / (kTile * kWarps);
  if (n > by_length) n = by_length;
  return n < 1 ? 1 : (n > kMaxSplit ? kMaxSplit : n);
}

}  // namespace

size_t decode_attention_scratch_bytes(int batch, int hkv, int head_dim, int s_max, int* n_split_out) {
  const int n_split = splits_for(batch * hkv, s_max);
  if (n_split_out) *n_split_out = n_split;
  const size_t partials = (size_t)batch * hkv * n_split * kHeads * (head_dim + 2) * sizeof(float);
  return 256 + ((size_t)batch * hkv * sizeof(unsigned int) + 255) / 256 * 256 + partials;
}

int launch_decode_attention(const void* qkv, void* k_cache, void* v_cache, void* out, void* scratch,
                            size_t scratch_bytes, int batch, int hq, int hkv, int head_dim, int s_max, int pos0,
                            const int* pos_dev, float rope_theta, cudaStream_t stream) {
  if (rope_theta != 0.f && rope_theta <= 1.0f) return cudaErrorInvalidValue;
  const float log2_theta = rope_theta != 0.f ? log2f(rope_theta) : 0.f;
  if (batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || hq / hkv > kHeads || (head_dim != 64 && head_dim != 128) ||
      s_max < 1 || (pos_dev == nullptr && (pos0 < 0 || pos0 >= s_max)))
    return cudaErrorInvalidValue;
  if (!aligned16(qkv) || !aligned16(k_cache) || !aligned16(v_cache) || !aligned16(out) || !aligned16(scratch))
    return cudaErrorInvalidValue;
  int n_split = 1;
  if (decode_attention_scratch_bytes(batch, hkv, head_dim, s_max, &n_split) > scratch_bytes) return cudaErrorInvalidValue;
  // layout of the scratch: [0, 256) unused, then one arrival counter per (b, kv head) (zero between
  // launches: the combining CTA resets it), then the partials
  unsigned int* counters = reinterpret_cast<unsigned int*>(static_cast<char*>(scratch) + 256);
  const size_t counter_bytes = ((size_t)batch * hkv * sizeof(unsigned int) + 255) / 256 * 256;
  float* partials = reinterpret_cast<float*>(static_cast<char*>(scratch) + 256 + counter_bytes);
  const float scale = 1.4426950408889634f / sqrtf((float)head_dim);          // scores in units of log2
  const dim3 grid((unsigned)(batch * hkv), (unsigned)n_split);
  auto q = static_cast<const __nv_bfloat16*>(qkv);
  auto kc = static_cast<__nv_bfloat16*>(k_cache);
  auto vc = static_cast<__nv_bfloat16*>(v_cache);
  auto o = static_cast<__nv_bfloat16*>(out);
  if (head_dim == 128)
    decode_attention_kernel<128><<<grid, kWarps * 32, 0, stream>>>(q, kc, vc, o, partials, counters, hq, hkv, s_max, pos0,
                                                                   pos_dev, scale, log2_theta);
  else
    decode_attention_kernel<64><<<grid, kWarps * 32, 0, stream>>>(q, kc, vc, o, partials, counters, hq, hkv, s_max, pos0,
                                                                  pos_dev, scale, log2_theta);
  return (int)cudaGetLastError();
}

}  // namespace smr
