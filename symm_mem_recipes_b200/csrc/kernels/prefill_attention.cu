// Causal attention over a short prompt, for the prefill of a world of one.  No upstream counterpart.
//
//     out[b, s, h, :] = softmax(q k^T / sqrt(D)) v        q, k, v rotated, in rows of the QKV projection
//
// What bounds it: latency.  A prompt of a few hundred tokens is under 1 GFLOP of attention and its keys and values
// fit in L2 many times over; a tiled flash kernel gives 32 CTAs to it and walks the keys one tile after the
// other (509 tokens x 8 heads: 13 us with PyTorch's, whose call also costs the host 20 us and cannot start under
// its predecessor).  Here a CTA takes 16 queries of one head and its four warps take the 16-key tiles in turns,
// so that no warp sees more than S / 64 tiles; their results meet in shared memory.  The arithmetic is that
// of decode_attention.cuh with all 16 rows of the MMA in use: K and V go from global memory straight into fragment
// registers, the next tile's K while this one's softmax runs.
//
// Every CTA reads its keys and values by itself, about S / 2 x 4 D bytes out of L2, so the traffic grows with
// batch x heads x S^2 / 16 and a kernel that shares tiles through shared memory wins on long prompts: see
// prefill_attention_preferred.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../device/pdl.cuh"
#include "../device/vec.cuh"
#include "decode_attention.cuh"
#include "launch.h"
#include "residency.h"

namespace smr {

namespace {

constexpr int kRows = 16;          // queries of a CTA
constexpr int kKeys = 16;          // keys of a tile
constexpr int kWarps = 4;

template <int D>
__global__ void __launch_bounds__(kWarps * 32, 2)
prefill_attention_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ out, int seq, int hq, int hkv,
                         float scale) {
  constexpr int NJ = D / 32, NI = D / 64, kPitch = D + 4;
  __shared__ __align__(16) float sm[kWarps][kRows][kPitch];
  __shared__ float2 ml[kWarps][kRows];                             // (max, sum)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int qb = (int)gridDim.x - 1 - (int)blockIdx.x;             // the longest rows first
  const int b = (int)blockIdx.y / hq, h = (int)blockIdx.y - b * hq, kvh = h / (hq / hkv);
  const size_t pitch = (size_t)(hq + 2 * hkv) * D;
  const __nv_bfloat16* base = qkv + (size_t)b * seq * pitch;
  const __nv_bfloat16* kc = base + (size_t)(hq + kvh) * D;
  const __nv_bfloat16* vc = kc + (size_t)hkv * D;
  const int q0 = qb * kRows;

  attn::Tile<D> f;
  const Vec16 zero{0u, 0u, 0u, 0u};
  auto load_k = [&](int tile) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int p = tile * kKeys + u * 8 + g;
      const __nv_bfloat16* src = kc + (size_t)p * pitch + t * 8;
#pragma unroll
      for (int j = 0; j < NJ; ++j) f.k[u][j] = p < seq ? ld_16(src + j * 32) : zero;
    }
  };
  auto load_v = [&](int tile) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int p = tile * kKeys + 2 * t + (r & 1) + (r >> 1) * 8;
      const __nv_bfloat16* src = vc + (size_t)p * pitch + g * 8;
#pragma unroll
      for (int i = 0; i < NI; ++i) f.v[r][i] = p < seq ? ld_16(src + i * 64) : zero;
    }
  };

  pdl_launch_dependents();
  pdl_wait();
  if (warp <= qb) {
    load_k(warp);
    load_v(warp);
  }
  Vec16 q[2][NJ];                                                  // rows g and g + 8, dimensions 32 j + 8 t ..
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int p = q0 + u * 8 + g;
#pragma unroll
    for (int j = 0; j < NJ; ++j) q[u][j] = p < seq ? ld_16(base + (size_t)p * pitch + (size_t)h * D + j * 32 + t * 8) : zero;
  }

  float m_run[2] = {attn::kNoScore, attn::kNoScore}, l_run[2] = {0.f, 0.f};   // rows g and g + 8
  float acc[2][D / 16][4];                                         // O^T of rows 0..7 and 8..15, as attn::State
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int i = 0; i < D / 16; ++i) acc[u][i][0] = acc[u][i][1] = acc[u][i][2] = acc[u][i][3] = 0.f;

  for (int tile = warp; tile <= qb; tile += kWarps) {
    const int next = tile + kWarps;
    float s[2][4];                                                 // keys 8 u + 2 t, + 1 of row g, then of row g + 8
#pragma unroll
    for (int u = 0; u < 2; ++u) s[u][0] = s[u][1] = s[u][2] = s[u][3] = 0.f;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        attn::mma_16816(s[u], q[0][j].x, q[1][j].x, q[0][j].y, q[1][j].y, f.k[u][j].x, f.k[u][j].y);
        attn::mma_16816(s[u], q[0][j].z, q[1][j].z, q[0][j].w, q[1][j].w, f.k[u][j].z, f.k[u][j].w);
      }
    if (next <= qb) load_k(next);                                  // into the registers the first MMA has read
    uint32_t prob[2][2];                                           // [rows 0..7 / 8..15][key octet]
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float mx = attn::kNoScore;
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float& x = s[u][2 * r + e];
          // only the last tile, the one the queries are in, has keys beyond them
          x = tile < qb || u * 8 + 2 * t + e <= r * 8 + g ? x * scale : attn::kNoScore;
          mx = fmaxf(mx, x);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run[r], mx);
      if (__any_sync(0xffffffffu, m_new > m_run[r])) {
        const float corr = exp2f(m_run[r] - m_new);
        l_run[r] *= corr;
        const float c0 = __shfl_sync(0xffffffffu, corr, 8 * t), c1 = __shfl_sync(0xffffffffu, corr, 8 * t + 4);
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
          acc[r][i][0] *= c0; acc[r][i][1] *= c1;
          acc[r][i][2] *= c0; acc[r][i][3] *= c1;
        }
        m_run[r] = m_new;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float p0 = exp2f(s[u][2 * r] - m_run[r]), p1 = exp2f(s[u][2 * r + 1] - m_run[r]);   // 0 where masked
        l_run[r] += p0 + p1;
        prob[r][u] = pack_bf16x2(p0, p1);
      }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int w = 0; w < 4; ++w) {                                // word w: dimensions 64 i + 8 g + 2 w, + 1
        const uint32_t r0 = (&f.v[0][i].x)[w], r1 = (&f.v[1][i].x)[w];
        const uint32_t r2 = (&f.v[2][i].x)[w], r3 = (&f.v[3][i].x)[w];
        const uint32_t a0 = __byte_perm(r0, r1, 0x5410), a1 = __byte_perm(r0, r1, 0x7632);
        const uint32_t a2 = __byte_perm(r2, r3, 0x5410), a3 = __byte_perm(r2, r3, 0x7632);
        attn::mma_16816(acc[0][i * 4 + w], a0, a1, a2, a3, prob[0][0], prob[0][1]);
        attn::mma_16816(acc[1][i * 4 + w], a0, a1, a2, a3, prob[1][0], prob[1][1]);
      }
    if (next <= qb) load_v(next);
  }

  // ---- the four warps meet ----
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    if (t == 0) ml[warp][r * 8 + g] = make_float2(m_run[r], l_run[r]);
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) {                                // four dimensions of query 8 r + 2 t + (c & 1)
        const int u = c & 1, at = i * 4 + (c & 2);
        *reinterpret_cast<float4*>(&sm[warp][r * 8 + 2 * t + u][i * 64 + g * 8 + 2 * (c & 2)]) =
            make_float4(acc[r][at][u], acc[r][at][u + 2], acc[r][at + 1][u], acc[r][at + 1][u + 2]);
      }
  }
  __syncthreads();
  constexpr int kPer = D / 32;                                     // consecutive dimensions of a lane
#pragma unroll
  for (int r = warp * (kRows / kWarps); r < (warp + 1) * (kRows / kWarps); ++r) {
    if (q0 + r >= seq) break;
    float big = attn::kNoScore, sum = 0.f, a[kPer];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) big = fmaxf(big, ml[w][r].x);
#pragma unroll
    for (int d = 0; d < kPer; ++d) a[d] = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float fw = exp2f(ml[w][r].x - big);                    // 0 for a warp without a tile
      sum += fw * ml[w][r].y;
#pragma unroll
      for (int d = 0; d < kPer; ++d) a[d] += fw * sm[w][r][lane * kPer + d];
    }
    const float inv = 1.0f / sum;
    uint32_t o[kPer / 2];
#pragma unroll
    for (int d = 0; d < kPer / 2; ++d) o[d] = pack_bf16x2(a[2 * d] * inv, a[2 * d + 1] * inv);
    __nv_bfloat16* dst = out + ((size_t)b * seq + q0 + r) * ((size_t)hq * D) + (size_t)h * D + lane * kPer;
    if constexpr (kPer == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
    else *reinterpret_cast<uint32_t*>(dst) = o[0];
  }
}

}  // namespace

// Against PyTorch's (device times, us; its call costs another 4 of gaps before and after it, because it neither starts
// under its predecessor nor lets its successor start, and 20 of host time that short prompts do not hide):
//     batch x tokens (8 heads, D 128)   1 x 64  1 x 300  1 x 509  4 x 200  8 x 128  2 x 509  4 x 300  16 x 128  8 x 300
//     here                                 3.3      7.3     10.8      9.3      8.4     17.2     14.1      14.3     23.7
//     there                                3.8     11.6     13.3     10.8      4.9     13.4     12.5       7.2     12.9
// The line lies at two waves of CTAs (two per SM) and at 48 MB read from L2.
bool prefill_attention_preferred(int batch, int seq, int hq, int hkv, int head_dim) {
  if ((head_dim != 64 && head_dim != 128) || hkv < 1 || hq % hkv != 0) return false;
  const double ctas = (double)batch * hq * ((seq + kRows - 1) / kRows), read = (double)batch * hq * seq * seq / 8.0 * head_dim;
  return ctas <= 4.0 * device_sms() && read <= 48.0e6;
}

int launch_prefill_attention(const void* qkv, void* out, int batch, int seq, int hq, int hkv, int head_dim, cudaStream_t stream) {
  if (batch < 1 || seq < 1 || hkv < 1 || hq % hkv != 0 || (head_dim != 64 && head_dim != 128) ||
      (long long)batch * hq > 65535 || ((uintptr_t)qkv | (uintptr_t)out) % 16 != 0)
    return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((seq + kRows - 1) / kRows), (unsigned)(batch * hq));
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const float scale = 1.4426950408889634f / sqrtf((float)head_dim);            // scores in units of log2
  const auto* in = static_cast<const __nv_bfloat16*>(qkv);
  auto* o = static_cast<__nv_bfloat16*>(out);
  return (int)(head_dim == 128 ? cudaLaunchKernelEx(&cfg, prefill_attention_kernel<128>, in, o, seq, hq, hkv, scale)
                               : cudaLaunchKernelEx(&cfg, prefill_attention_kernel<64>, in, o, seq, hq, hkv, scale));
}

}  // namespace smr
