// Attention of one decode step (one new token per sequence) for this rank's heads, split along the cached
// sequence ("flash decoding").  No upstream counterpart (the upstream recipes stop at the single fused op).
//
//     out[b, h, :] = softmax(q[b, h] . K[b, 0..pos, h / G] / sqrt(D)) V[b, 0..pos, h / G]      G = hq / hkv
//
// What bounds it: the cache crosses HBM once (2 * D * 2 bytes per position and KV head); with a short
// context, the chain of dependent steps from the launch to the merged result.
//   * The G <= 8 query heads of a KV head are one MMA operand (mma.sync m16n8k16): S = Q K^T takes the heads
//     as M (rows G..15 are zero) and 8 positions as N; O^T = V^T P^T takes 16 dimensions as M and the heads as
//     N.  With that pairing the scores leave the first MMA in exactly the registers the second one reads
//     them from, and both K and V go from global memory straight into fragment registers with 16-byte
//     loads: the order of the dimensions inside a fragment is free as long as both operands agree, so a
//     lane takes eight consecutive dimensions.  No shared memory, no transposition, no barrier in the
//     loop.  (tcgen05 would pad 8 heads to 128 rows and need the probabilities written back to shared
//     memory; the tensor work here is under 2 % of the time.)
//   * The probabilities enter the second MMA as a bf16 pair, P = hi + lo (two MMAs): the weighted sum keeps
//     fp32-grade weights.
//   * A warp takes 16 positions at a time; the next K (4 KB at D = 128) is loaded into the registers that the
//     first MMA has read, the next V into those of the second.  Sixteen warps an SM (two CTAs) keep
//     64-128 KB in flight.  Tiles are dealt out so that neighbouring tiles go to different CTAs: a short
//     context still uses every SM.
//   * The warps of a CTA merge through shared memory, the CTAs of a (sequence, KV head) through scratch
//     memory: the last one to arrive adds the others up.
// The new token's key and value come from the QKV row (its warp also writes them into the caches), so no CTA
// depends on another's cache write.  The position may come from device memory and the grid does not depend
// on it: a captured graph serves every position.  In a decode chain the kernel is launched with programmatic
// stream serialization: rotation angles and the first tiles are loaded before griddepcontrol.wait.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../device/pdl.cuh"
#include "../device/vec.cuh"
#include "launch.h"

namespace smr {

namespace {

constexpr int kWarps = 8;
constexpr int kHeads = 8;               // query heads per KV head at most (the MMA's N)
constexpr int kTile = 16;               // positions a warp takes at a time
constexpr int kMaxSplit = 64;           // CTAs per (sequence, KV head) at most
// "No position seen yet" as a running maximum.  A finite stand-in for minus infinity: a warp or a CTA may see
// no position at all, and exp(-inf - (-inf)) would be NaN in the merges, while exp(kNoScore - kNoScore) = 1
// weights a sum and a vector that are both zero.
constexpr float kNoScore = -1.0e30f;

// D[16 x 8] += A[16 x 16] B[16 x 8], bf16 in, fp32 out
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A warp's 16 positions of K and V.  Lane (g = lane / 4, t = lane % 4) holds
//   K: positions g and g + 8, dimensions 32 j + 8 t .. + 7
//   V: positions 2t, 2t + 1, 2t + 8, 2t + 9, dimensions 64 i + 8 g .. + 7
template <int D>
struct Tile {
  Vec16 k[2][D / 32];
  Vec16 v[4][D / 64];
};

template <int D>
__global__ void __launch_bounds__(kWarps * 32, 2)
decode_attention_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache,
                        __nv_bfloat16* __restrict__ out, float* scratch, unsigned int* counters, int hq, int hkv,
                        int s_max, int pos0, const int* __restrict__ pos_dev, float scale, float log2_theta) {
  constexpr int kRow = D + 2;                                  // D weighted-V sums, then max and sum
  constexpr int NJ = D / 32, NI = D / 64;                      // 16-byte loads of a K row, of a V row
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
  pdl_launch_dependents();
  int pos = pos_dev != nullptr ? *pos_dev : pos0;
  pos = pos < 0 ? 0 : (pos >= s_max ? s_max - 1 : pos);
  // tile 0 is the new token, tiles 1.. are the cached positions
  const int n_tiles = 1 + (pos + kTile - 1) / kTile;
  const size_t pitch = (size_t)hkv * D;                        // elements between positions
  __nv_bfloat16* kc = k_cache + ((size_t)b * s_max * hkv + kvh) * D;
  __nv_bfloat16* vc = v_cache + ((size_t)b * s_max * hkv + kvh) * D;

  Tile<D> f;
  auto load_k = [&](int tile) {
    const int p0 = (tile - 1) * kTile;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int p = p0 + u * 8 + g;
      const __nv_bfloat16* src = kc + (size_t)p * pitch + t * 8;
#pragma unroll
      for (int j = 0; j < NJ; ++j) f.k[u][j] = p < pos ? ld_16_stream(src + j * 32) : Vec16{0u, 0u, 0u, 0u};
    }
  };
  auto load_v = [&](int tile) {
    const int p0 = (tile - 1) * kTile;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int p = p0 + 2 * t + (r & 1) + (r >> 1) * 8;
      const __nv_bfloat16* src = vc + (size_t)p * pitch + g * 8;
#pragma unroll
      for (int i = 0; i < NI; ++i) f.v[r][i] = p < pos ? ld_16_stream(src + i * 64) : Vec16{0u, 0u, 0u, 0u};
    }
  };

  if (unit > 0 && unit < n_tiles) {
    load_k(unit);
    load_v(unit);
  }

  // Rotation of the new token's queries and key (log2_theta != 0): the pair (i, i + D/2) sits in loads j and
  // j + NJ/2 of the same lane.  Results are rounded to bf16 as the stand-alone RoPE kernel rounds them.
  // The angles are the same for every head: D / 2 threads compute them once per CTA.
  const bool rotate = log2_theta != 0.f;
  if (rotate) {
    const int i = threadIdx.x;
    if (i < D / 2) {
      float ang = (float)pos * exp2f(-(2.0f * (float)i / (float)D) * log2_theta);
      ang -= 6.283185307179586f * rintf(ang * 0.15915494309189535f);
      __sincosf(ang, &angles[i].y, &angles[i].x);
    }
    __syncthreads();
  }
  auto rope = [&](Vec16 (&x)[NJ]) {
#pragma unroll
    for (int j = 0; j < NJ / 2; ++j) {
      uint32_t* lo = &x[j].x;
      uint32_t* hi = &x[j + NJ / 2].x;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float a0 = bf16lo_to_f32(lo[w]), a1 = bf16hi_to_f32(lo[w]);
        const float b0 = bf16lo_to_f32(hi[w]), b1 = bf16hi_to_f32(hi[w]);
        const float4 cs = *reinterpret_cast<const float4*>(&angles[j * 32 + t * 8 + 2 * w]);   // cos, sin of two pairs
        lo[w] = pack_bf16x2(a0 * cs.x - b0 * cs.y, a1 * cs.z - b1 * cs.w);
        hi[w] = pack_bf16x2(b0 * cs.x + a0 * cs.y, b1 * cs.z + a1 * cs.w);
      }
    }
  };

  pdl_wait();
  const __nv_bfloat16* row = qkv + (size_t)b * (hq + 2 * hkv) * D;
  Vec16 q[NJ];                                                 // head g, dimensions 32 j + 8 t ..
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    q[j] = g < G ? ld_16(row + (size_t)(kvh * G + g) * D + j * 32 + t * 8) : Vec16{0u, 0u, 0u, 0u};

  // The new token is a tile of one position: lanes g = 0 hold its key, lanes t = 0 its value, the rest is zero.
  if (unit == 0) {
    const Vec16 zero{0u, 0u, 0u, 0u};
    const __nv_bfloat16* k_new = row + (size_t)(hq + kvh) * D;
    const __nv_bfloat16* v_new = row + (size_t)(hq + hkv + kvh) * D;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      f.k[0][j] = g == 0 ? ld_16(k_new + j * 32 + t * 8) : zero;
      f.k[1][j] = zero;
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      f.v[0][i] = t == 0 ? ld_16(v_new + i * 64 + g * 8) : zero;
      f.v[1][i] = f.v[2][i] = f.v[3][i] = zero;
    }
    if (rotate) rope(f.k[0]);
    __nv_bfloat16* kd = kc + (size_t)pos * pitch;
    __nv_bfloat16* vd = vc + (size_t)pos * pitch;
    if (g == 0) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) st_16(kd + j * 32 + t * 8, f.k[0][j]);
    }
    if (t == 0) {
#pragma unroll
      for (int i = 0; i < NI; ++i) st_16(vd + i * 64 + g * 8, f.v[0][i]);
    }
  }
  if (rotate) rope(q);

  // Running state: maximum of head g in units of log2 (the same in its four lanes), this lane's share of the
  // sum, and O^T: acc[m] holds dimensions dim(m, 0) (c0, c1) and dim(m, 1) (c2, c3) of heads 2t and 2t + 1.
  float m_run = kNoScore, l_run = 0.f;
  float acc[D / 16][4];
#pragma unroll
  for (int m = 0; m < D / 16; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;

  for (int i = unit; i < n_tiles; i += n_units) {
    const int n_valid = i == 0 ? 1 : pos - (i - 1) * kTile, next = i + n_units;
    float s[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      s[u][0] = s[u][1] = s[u][2] = s[u][3] = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        mma_16816(s[u], q[j].x, 0u, q[j].y, 0u, f.k[u][j].x, f.k[u][j].y);
        mma_16816(s[u], q[j].z, 0u, q[j].w, 0u, f.k[u][j].z, f.k[u][j].w);
      }
    }
    if (next < n_tiles) load_k(next);                          // into the registers the first MMA has read
    float mx = kNoScore;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[u][e] = u * 8 + 2 * t + e < n_valid ? s[u][e] * scale : kNoScore;
        mx = fmaxf(mx, s[u][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx);
    if (__any_sync(0xffffffffu, m_new > m_run)) {
      const float corr = exp2f(m_run - m_new);
      l_run *= corr;
      const float c0 = __shfl_sync(0xffffffffu, corr, 8 * t), c1 = __shfl_sync(0xffffffffu, corr, 8 * t + 4);
#pragma unroll
      for (int m = 0; m < D / 16; ++m) {
        acc[m][0] *= c0; acc[m][1] *= c1;
        acc[m][2] *= c0; acc[m][3] *= c1;
      }
      m_run = m_new;
    }
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float p0 = s[u][0] > 0.5f * kNoScore ? exp2f(s[u][0] - m_run) : 0.f;
      const float p1 = s[u][1] > 0.5f * kNoScore ? exp2f(s[u][1] - m_run) : 0.f;
      l_run += p0 + p1;
      hi[u] = pack_bf16x2(p0, p1);
      lo[u] = pack_bf16x2(p0 - bf16lo_to_f32(hi[u]), p1 - bf16hi_to_f32(hi[u]));
    }
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int w = 0; w < 4; ++w) {                            // word w: dimensions 64 i + 8 g + 2 w, + 1
        const uint32_t r0 = (&f.v[0][i].x)[w], r1 = (&f.v[1][i].x)[w];
        const uint32_t r2 = (&f.v[2][i].x)[w], r3 = (&f.v[3][i].x)[w];
        const uint32_t a0 = __byte_perm(r0, r1, 0x5410), a1 = __byte_perm(r0, r1, 0x7632);
        const uint32_t a2 = __byte_perm(r2, r3, 0x5410), a3 = __byte_perm(r2, r3, 0x7632);
        mma_16816(acc[i * 4 + w], a0, a1, a2, a3, hi[0], hi[1]);
        mma_16816(acc[i * 4 + w], a0, a1, a2, a3, lo[0], lo[1]);
      }
    if (next < n_tiles) load_v(next);
  }

  // ---- the CTA's warps merge through shared memory into one partial per CTA ----
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
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
  int n = 296 / (rows > 0 ? rows : 1);
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
                            const int* pos_dev, float rope_theta, cudaStream_t stream, bool overlap) {
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
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(batch * hkv), (unsigned)n_split);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  auto q = static_cast<const __nv_bfloat16*>(qkv);
  auto kc = static_cast<__nv_bfloat16*>(k_cache);
  auto vc = static_cast<__nv_bfloat16*>(v_cache);
  auto o = static_cast<__nv_bfloat16*>(out);
  return (int)(head_dim == 128
                   ? cudaLaunchKernelEx(&cfg, decode_attention_kernel<128>, q, kc, vc, o, partials, counters, hq, hkv,
                                        s_max, pos0, pos_dev, scale, log2_theta)
                   : cudaLaunchKernelEx(&cfg, decode_attention_kernel<64>, q, kc, vc, o, partials, counters, hq, hkv,
                                        s_max, pos0, pos_dev, scale, log2_theta));
}

}  // namespace smr
