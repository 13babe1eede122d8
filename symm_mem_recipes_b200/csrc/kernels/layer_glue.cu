// Rank-local pieces of a Llama-style decoder layer that sit between the fused
// GEMM + collective kernels: RMSNorm (optionally fused with the residual add
// that precedes it), rotary embedding in place on the QKV buffer, and
// SiLU(gate) * up.  Each is one pass over its operand in bf16 with fp32 math;
// the PyTorch compositions they replace take five to ten passes with fp32
// temporaries.  No upstream counterpart (the upstream recipes stop at the
// single fused op).
//
// Arithmetic contracts (what the CPU oracles in oracle/cpu_reference.cpp and
// the tests pin down):
//   rms_norm:  s = x (+ r, rounded to bf16 when r is given; also stored as
//              `sum_out`);  n = bf16( s * rsqrt(mean(s^2) + eps) );
//              out = bf16( n * w ).
//   rope:      pairs (i, i + D/2) of every rotated head, Llama convention:
//              angle = pos * theta^(-2i/D), fp32; results rounded to bf16.
//   silu_mul:  out = bf16( g / (1 + exp(-g)) * u ) for gate g, up u.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../device/pdl.cuh"
#include "../device/vec.cuh"
#include "launch.h"
#include "residency.h"

namespace smr {

namespace {

__device__ __forceinline__ void unpack8(const Vec16& v, float (&f)[8]) {
  f[0] = bf16lo_to_f32(v.x); f[1] = bf16hi_to_f32(v.x);
  f[2] = bf16lo_to_f32(v.y); f[3] = bf16hi_to_f32(v.y);
  f[4] = bf16lo_to_f32(v.z); f[5] = bf16hi_to_f32(v.z);
  f[6] = bf16lo_to_f32(v.w); f[7] = bf16hi_to_f32(v.w);
}
__device__ __forceinline__ Vec16 pack8(const float (&f)[8]) {
  Vec16 o;
  o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
  return o;
}
__device__ __forceinline__ float round_bf16(float f) {
  return __bfloat162float(__float2bfloat16_rn(f));
}

// A CTA takes rows blockIdx.x, blockIdx.x + gridDim.x, ...; a row lives in registers (VPT vectors of eight per thread):
// x and the residual are read once, s and the result written once, and the next row is loaded before this one is
// reduced, so that the reduction's latency is not a hole in the memory stream.  The weight stays in registers.
// Bound by HBM for a prefill (32768 x 8192: 235 us with a second pass over the row; 1.07 GB are 164 us at
// the measured copy rate), by latency for a handful of rows, which is why a row is spread over up to 1024
// threads there.  `sum_out` may be the buffer of `x` or of `residual` (running residual stream
// updated in place) and `out` may be the buffer of `x`; `out` must not be the
// buffer of `sum_out` or of `residual`.
template <int THREADS, int VPT, bool kResidual>
__global__ void __launch_bounds__(THREADS, THREADS > 256 ? 1 : (VPT <= 2 ? 4 : (VPT == 4 && !kResidual ? 3 : (VPT == 4 ? 2 : 1))))
rms_norm_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual, const __nv_bfloat16* __restrict__ w,
                __nv_bfloat16* sum_out, __nv_bfloat16* out, int rows, int H, float eps) {
  pdl_launch_dependents();
  const int n_vec = H / 8;
  Vec16 g[VPT], s[VPT], r[kResidual ? VPT : 1];
  pdl_wait();
#pragma unroll
  for (int j = 0; j < VPT; ++j)
    g[j] = threadIdx.x + j * THREADS < n_vec ? ld_16(reinterpret_cast<const Vec16*>(w) + threadIdx.x + j * THREADS)
                                             : Vec16{0u, 0u, 0u, 0u};
  auto fetch = [&](int row) {
    const Vec16* xr = reinterpret_cast<const Vec16*>(x + (size_t)row * H);
    const Vec16* rr = reinterpret_cast<const Vec16*>(residual + (size_t)row * H);
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      s[j] = i < n_vec ? ld_16_stream(xr + i) : Vec16{0u, 0u, 0u, 0u};
      if constexpr (kResidual) r[j] = i < n_vec ? ld_16_stream(rr + i) : Vec16{0u, 0u, 0u, 0u};
    }
  };
  __shared__ float warp_sums[2][THREADS / 32];
  int parity = 0;
  fetch(blockIdx.x);
  for (int row = blockIdx.x; row < rows; row += gridDim.x, parity ^= 1) {
    Vec16 v[VPT];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      v[j] = s[j];
      if constexpr (kResidual) {
        v[j] = add_bf16x8(v[j], r[j]);
        const int i = threadIdx.x + j * THREADS;
        if (i < n_vec && sum_out != nullptr) st_16(reinterpret_cast<Vec16*>(sum_out + (size_t)row * H) + i, v[j]);
      }
      float a[8];
      unpack8(v[j], a);
#pragma unroll
      for (int q = 0; q < 8; ++q) ss += a[q] * a[q];
    }
    if (row + (int)gridDim.x < rows) fetch(row + gridDim.x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) warp_sums[parity][threadIdx.x >> 5] = ss;
    __syncthreads();
    float t = (threadIdx.x & 31) < THREADS / 32 ? warp_sums[parity][threadIdx.x & 31] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const float scale = rsqrtf(t / (float)H + eps);
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      float a[8], b[8];
      unpack8(v[j], a);
      unpack8(g[j], b);
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = round_bf16(a[q] * scale) * b[q];
      if (i < n_vec) st_16(reinterpret_cast<Vec16*>(out + (size_t)row * H) + i, pack8(a));
    }
  }
}

// Rows too long for registers (H > 16384): one CTA per row, two passes.  Pass 2 re-reads s (from L1 / L2).
__global__ void __launch_bounds__(256)
rms_norm_long_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual, const __nv_bfloat16* __restrict__ w,
                     __nv_bfloat16* sum_out, __nv_bfloat16* out, int H, float eps) {
  const size_t row = blockIdx.x;
  const Vec16* xr = reinterpret_cast<const Vec16*>(x + row * H);
  const Vec16* rr = residual ? reinterpret_cast<const Vec16*>(residual + row * H) : nullptr;
  Vec16* sr = sum_out ? reinterpret_cast<Vec16*>(sum_out + row * H) : nullptr;
  const int n_vec = H / 8;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n_vec; i += 256) {
    Vec16 v = ld_16(xr + i);
    if (rr != nullptr) v = add_bf16x8(v, ld_16(rr + i));
    if (sr != nullptr) st_16(sr + i, v);
    float a[8];
    unpack8(v, a);
#pragma unroll
    for (int q = 0; q < 8; ++q) ss += a[q] * a[q];
  }
  __shared__ float warp_sums[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = ss;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += warp_sums[i];
  const float scale = rsqrtf(t / (float)H + eps);
  for (int i = threadIdx.x; i < n_vec; i += 256) {
    // this thread stored s[i] itself in pass 1; reading it back (instead of x and r again) also
    // keeps the kernel correct when sum_out is the same buffer as x or as the residual
    Vec16 v = ld_16(sr != nullptr ? sr + i : xr + i);
    if (sr == nullptr && rr != nullptr) v = add_bf16x8(v, ld_16(rr + i));
    float a[8], g[8];
    unpack8(v, a);
    unpack8(ld_16(reinterpret_cast<const Vec16*>(w) + i), g);
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = round_bf16(a[q] * scale) * g[q];
    st_16(reinterpret_cast<Vec16*>(out + row * H) + i, pack8(a));
  }
}

// In place on rows of `row_stride` elements: heads [0, n_heads) of D elements
// each are rotated.  Token t sits at position pos0 + (t % seq); with `pos_dev`
// the first position is read from device memory instead (a decode step
// captured in a CUDA graph takes its position from a tensor).
// With caches ([tokens / seq, s_max, hkv, D] each) the last hkv of the rotated heads are also written to the key cache
// and the hkv heads after them to the value cache, at the token's place in its sequence.
// A warp takes a token: its first loads go out, then its angles are computed once into shared memory (a sine and cosine
// per pair instead of one per pair and head), then a lane rotates eight pairs of a head at a time.  The table is stored
// by [pair of the eight][eight], because the lanes of a head read the same pair of neighbouring eights: in the order of
// the pairs that was a 4-way bank conflict, as much time as the memory.  Four CTAs per SM need 64 registers.  Cold, 9 heads x
// 128: 16384 tokens 24.7 us with the conflicts, 22.5 at three CTAs, 20.5 now; 4096 tokens 12.3, 11.1, 10.3; one angle per
// pair and head 20.6 and 10.3, but 120 against 100 us for 72 heads of 16384 tokens, and two passes more for the caches.
__global__ void __launch_bounds__(256, 4)
rope_kernel(__nv_bfloat16* __restrict__ qkv, long long tokens, int row_stride, int n_heads, int D, int seq, int pos0,
            const int* __restrict__ pos_dev, float log2_theta, __nv_bfloat16* __restrict__ k_cache,
            __nv_bfloat16* __restrict__ v_cache, int s_max, int hkv) {
  extern __shared__ float2 angles[];                    // [warps][D / 2] (cos, sin)
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = D / 2;
  const long long t = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
  pdl_wait();
  if (t >= tokens) return;
  if (pos_dev != nullptr) pos0 = *pos_dev;
  const long long in_batch = t / seq;
  const int in_seq = (int)(t - in_batch * seq);
  const int vecs = D / 16;                              // items of eight pairs per head
  const int n_items = (n_heads + (v_cache != nullptr ? hkv : 0)) * vecs;
  __nv_bfloat16* row = qkv + t * row_stride;
  const size_t cache_row = ((size_t)in_batch * s_max + in_seq) * hkv;   // the token's row of a cache, in heads
  constexpr int kPer = 3;                               // a lane's items in flight: a row of 12 heads of 128 in one go
  Vec16 lo[kPer], hi[kPer];
  int head[kPer], v[kPer];
  auto load = [&](int item0) {
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int item = item0 + 32 * u;
      head[u] = item / vecs;
      v[u] = (item - head[u] * vecs) * 8;
      if (item < n_items) {
        lo[u] = ld_16_stream(row + (size_t)head[u] * D + v[u]);
        hi[u] = ld_16_stream(row + (size_t)head[u] * D + half + v[u]);
      }
    }
  };
  load(lane);
  float2* mine = angles + warp * half;
  for (int i = lane; i < half; i += 32) {               // pair index in [0, D/2)
    const float inv_freq = exp2f(-(2.0f * (float)i / (float)D) * log2_theta);
    float ang = (float)(pos0 + in_seq) * inv_freq;
    // bring the angle into [-pi, pi] before the fast sine / cosine
    ang -= 6.283185307179586f * rintf(ang * 0.15915494309189535f);
    float sn, cs;
    __sincosf(ang, &sn, &cs);
    mine[(i & 7) * vecs + (i >> 3)] = make_float2(cs, sn);
  }
  __syncwarp();
  for (int item0 = lane; item0 < n_items; item0 += 32 * kPer) {
    if (item0 != lane) load(item0);
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (item0 + 32 * u >= n_items) continue;
      if (head[u] >= n_heads) {                         // a value head: only copied
        __nv_bfloat16* dst = v_cache + (cache_row + (head[u] - n_heads)) * D + v[u];
        st_16(dst, lo[u]);
        st_16(dst + half, hi[u]);
        continue;
      }
      float x1[8], x2[8], y1[8], y2[8];
      unpack8(lo[u], x1);
      unpack8(hi[u], x2);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float2 c = mine[q * vecs + (v[u] >> 3)];
        y1[q] = x1[q] * c.x - x2[q] * c.y;
        y2[q] = x2[q] * c.x + x1[q] * c.y;
      }
      const Vec16 o1 = pack8(y1), o2 = pack8(y2);
      __nv_bfloat16* src = row + (size_t)head[u] * D + v[u];
      st_16(src, o1);
      st_16(src + half, o2);
      if (k_cache != nullptr && head[u] >= n_heads - hkv) {
        __nv_bfloat16* dst = k_cache + (cache_row + (head[u] - (n_heads - hkv))) * D + v[u];
        st_16(dst, o1);
        st_16(dst + half, o2);
      }
    }
  }
}

// gu [T, 2F]: gate = columns [0, F), up = [F, 2F); out [T, F].
__global__ void silu_mul_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                long long n_vec, int F) {
  const int vec_per_row = F / 8;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n_vec; idx += stride) {
    const long long row = idx / vec_per_row;
    const int cv = (int)(idx - row * vec_per_row);
    const __nv_bfloat16* g = gu + row * 2 * F + cv * 8;
    float a[8], b[8];
    unpack8(ld_16_stream(g), a);
    unpack8(ld_16_stream(g + F), b);
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = a[q] / (1.0f + __expf(-a[q])) * b[q];
    st_16(out + row * F + cv * 8, pack8(a));
  }
}

int grid_for(long long items, int threads, int num_sms) {
  long long blocks = (items + threads - 1) / threads;
  const long long cap = (long long)num_sms * 8;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

int launch_rms_norm(const void* x, const void* residual, const void* w, void* sum_out, void* out, int rows, int H,
                    float eps, cudaStream_t stream) {
  if (rows < 0 || H <= 0 || H % 8 != 0) return cudaErrorInvalidValue;
  if (!aligned16(x) || !aligned16(w) || !aligned16(out) || (residual && !aligned16(residual)) ||
      (sum_out && !aligned16(sum_out)))
    return cudaErrorInvalidValue;
  if (sum_out != nullptr && residual == nullptr) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const int n_vec = H / 8;
  const auto xb = static_cast<const __nv_bfloat16*>(x), rb = static_cast<const __nv_bfloat16*>(residual);
  const auto wb = static_cast<const __nv_bfloat16*>(w);
  const auto sb = static_cast<__nv_bfloat16*>(sum_out), ob = static_cast<__nv_bfloat16*>(out);
  if (n_vec > 2048) {
    rms_norm_long_kernel<<<rows, 256, 0, stream>>>(xb, rb, wb, sb, ob, H, eps);
    return (int)cudaGetLastError();
  }
  const int sms = device_sms();
  auto go = [&](auto kernel, int threads, int per_sm) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(rows < sms * per_sm ? rows : sms * per_sm));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, xb, rb, wb, sb, ob, rows, H, eps);
  };
  // fewer rows than SMs: one vector per thread, the shortest chain; else 256 threads, as many CTAs as the
  // registers of the widest rows allow per SM
  auto pick = [&](auto res) {
    constexpr bool R = decltype(res)::value;
    if (rows < sms && n_vec > 256 && n_vec <= 1024) return go(rms_norm_kernel<1024, 1, R>, 1024, 1);
    if (n_vec <= 256) return go(rms_norm_kernel<256, 1, R>, 256, 4);
    if (n_vec <= 512) return go(rms_norm_kernel<256, 2, R>, 256, 4);
    if (n_vec <= 1024) return go(rms_norm_kernel<256, 4, R>, 256, R ? 2 : 3);
    return go(rms_norm_kernel<256, 8, R>, 256, 1);
  };
  return residual != nullptr ? pick(std::true_type{}) : pick(std::false_type{});
}

int launch_rope_inplace(void* qkv, long long tokens, int row_stride, int n_heads, int head_dim, int seq, int pos0,
                        const int* pos_dev, float theta, cudaStream_t stream, void* k_cache, void* v_cache, int s_max,
                        int hkv) {
  if (tokens < 0 || n_heads < 1 || head_dim < 16 || head_dim % 16 != 0 || seq < 1 || row_stride % 8 != 0 ||
      (long long)n_heads * head_dim > row_stride || theta <= 1.0f || !aligned16(qkv))
    return cudaErrorInvalidValue;
  if ((k_cache == nullptr) != (v_cache == nullptr)) return cudaErrorInvalidValue;
  if (k_cache != nullptr &&
      (hkv < 1 || hkv > n_heads || (long long)(n_heads + hkv) * head_dim > row_stride || s_max < seq || tokens % seq != 0 ||
       pos_dev != nullptr || pos0 != 0 || !aligned16(k_cache) || !aligned16(v_cache)))
    return cudaErrorInvalidValue;
  if (tokens == 0) return cudaSuccess;
  int warps = 8;                                        // fewer where the tables of eight heads would not fit
  while (warps > 1 && (size_t)warps * (head_dim / 2) * sizeof(float2) > 48 * 1024) warps >>= 1;
  const size_t smem = (size_t)warps * (head_dim / 2) * sizeof(float2);
  if (smem > 48 * 1024) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((tokens + warps - 1) / warps));
  cfg.blockDim = dim3((unsigned)warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, rope_kernel, static_cast<__nv_bfloat16*>(qkv), tokens, row_stride, n_heads,
                                 head_dim, seq, pos0, pos_dev, log2f(theta), static_cast<__nv_bfloat16*>(k_cache),
                                 static_cast<__nv_bfloat16*>(v_cache), s_max, hkv);
}

int launch_silu_mul(const void* gate_up, void* out, long long rows, int F, int num_sms, cudaStream_t stream) {
  if (rows < 0 || F <= 0 || F % 8 != 0 || !aligned16(gate_up) || !aligned16(out)) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const long long n_vec = rows * (F / 8);
  silu_mul_kernel<<<grid_for(n_vec, 256, num_sms), 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(gate_up),
                                                                    static_cast<__nv_bfloat16*>(out), n_vec, F);
  return (int)cudaGetLastError();
}

}  // namespace smr
