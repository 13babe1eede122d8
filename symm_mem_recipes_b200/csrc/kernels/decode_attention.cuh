// The arithmetic of one decode step of attention, shared by the stand-alone kernel (decode_attention.cu) and the
// persistent decode step (decode_stack.cu): a warp's share of softmax(q K^T) V for the G <= 8 query heads of one KV head.
//
//   * The query heads are one MMA operand (mma.sync m16n8k16): S = Q K^T takes the heads as M (rows G..15 are
//     zero) and 8 positions as N; O^T = V^T P^T takes 16 dimensions as M and the heads as N.  With that
//     pairing the scores leave the first MMA in exactly the registers the second one reads them from, and
//     both K and V go from global memory straight into fragment registers with 16-byte loads: the order of
//     the dimensions inside a fragment is free as long as both operands agree, so a lane takes eight
//     consecutive dimensions.  No shared memory, no transposition, no barrier in the loop.  (tcgen05 would
//     pad 8 heads to 128 rows and need the probabilities written back to shared memory; the tensor work
//     here is under 2 % of the time.)
//   * The probabilities enter the second MMA as a bf16 pair, P = hi + lo (two MMAs): the weighted sum keeps
//     fp32-grade weights.
//   * A warp takes 16 positions at a time; the next K (4 KB at D = 128) is loaded into the registers that the
//     first MMA has read, the next V into those of the second.  Tiles are dealt out so that neighbouring
//     tiles go to different CTAs: a short context still uses every SM.
#pragma once
#include <cuda_bf16.h>

#include "../device/vec.cuh"

namespace smr {
namespace attn {

constexpr int kHeads = 8;               // query heads per KV head at most (the MMA's N)
constexpr int kTile = 16;               // positions a warp takes at a time
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

// A warp's result.  Lane (g, t): maximum (in units of log2) of head g, the same in its four lanes; its own share of the
// sum; O^T: acc[4 i + w] holds dimensions 64 i + 8 g + 2 w (c0, c1) and the next one (c2, c3) of heads 2t and 2t + 1.
template <int D>
struct State {
  float m, l;
  float acc[D / 16][4];
};

// (cos, sin) of the D / 2 pairs at `pos`, by the first D / 2 threads of a group; the caller synchronises.
template <int D>
__device__ __forceinline__ void fill_angles(float2* angles, int thread, int pos, float log2_theta) {
  if (thread < D / 2) {
    float ang = (float)pos * exp2f(-(2.0f * (float)thread / (float)D) * log2_theta);
    ang -= 6.283185307179586f * rintf(ang * 0.15915494309189535f);
    __sincosf(ang, &angles[thread].y, &angles[thread].x);
  }
}

// The cached positions of a tile into L2, a lane per 128 bytes.  The persistent step keeps two tiles a warp ahead: with one
// (in registers) a tile takes as long as HBM's latency under load, with six before the attention the requests of
// a long context crowd out the loads in front of them.  Two layers of a TP8 share as one step, us, 16 sequences at
//     position                             2000   4000   6000   8000
//     six before the attention, none in it 118.8  129.4  138.8  148.2
//     two before it                        118.8  126.1  133.5  142.9
//     and one more per tile in it          118.7  125.9  133.4  141.8   (the second next instead of the next: 143.6)
template <int D>
__device__ __forceinline__ void prefetch_tile(const __nv_bfloat16* kc, const __nv_bfloat16* vc, size_t pitch, int pos, int tile) {
  const int lane = threadIdx.x & 31, at = (tile - 1) * kTile + (D == 128 ? lane >> 1 : lane & 15);
  if (tile > 0 && at < pos) {
    const size_t off = (size_t)at * pitch + (D == 128 ? (lane & 1) * 64 : 0);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(kc + off));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(vc + off));
  }
}

// `kc`, `vc`: the caches at (sequence, KV head), `pitch` elements between positions.  Unit `unit` of `n_units` takes
// tiles unit, unit + n_units, ...; tile 0 is the new token (its unit also writes it into the caches), tiles 1.. are the
// cached positions [0, pos).  `row(part, head, d)` gives eight bf16 of the new token: part 0 query head, 1 key, 2 value.
// `angles`: the rotation of queries and key, or nullptr.  `ready()` is called between the first loads and the first row().
// `kAhead`: the tile after the next one into L2 (where weights come in at the same time; by itself the kernel of 16
// sequences at 6500 takes 22.6 us with it and 21.8 without).
template <int D, bool kAhead, class Ready, class Row>
__device__ __forceinline__ void attend(__nv_bfloat16* kc, __nv_bfloat16* vc, size_t pitch, int pos, int unit, int n_units,
                                       int G, float scale, const float2* angles, Ready ready, Row row, State<D>& st) {
  constexpr int NJ = D / 32, NI = D / 64;                      // 16-byte loads of a K row, of a V row
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n_tiles = 1 + (pos + kTile - 1) / kTile;
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
  ready();

  // the pair (i, i + D/2) sits in loads j and j + NJ/2 of the same lane; results are rounded to bf16 as the
  // stand-alone RoPE kernel rounds them
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

  Vec16 q[NJ];                                                 // head g, dimensions 32 j + 8 t ..
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    q[j] = g < G ? row(0, g, j * 32 + t * 8) : Vec16{0u, 0u, 0u, 0u};

  // The new token is a tile of one position: lanes g = 0 hold its key, lanes t = 0 its value, the rest is zero.
  if (unit == 0) {
    const Vec16 zero{0u, 0u, 0u, 0u};
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      f.k[0][j] = g == 0 ? row(1, 0, j * 32 + t * 8) : zero;
      f.k[1][j] = zero;
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      f.v[0][i] = t == 0 ? row(2, 0, i * 64 + g * 8) : zero;
      f.v[1][i] = f.v[2][i] = f.v[3][i] = zero;
    }
    if (angles != nullptr) rope(f.k[0]);
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
  if (angles != nullptr) rope(q);

  float& m_run = st.m;
  float& l_run = st.l;
  auto& acc = st.acc;
  m_run = kNoScore;
  l_run = 0.f;
#pragma unroll
  for (int m = 0; m < D / 16; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;

  for (int i = unit; i < n_tiles; i += n_units) {
    const int n_valid = i == 0 ? 1 : pos - (i - 1) * kTile, next = i + n_units;
    float s[2][4], s2[2][4];                                   // two chains each: an MMA waits for the one before it
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      s[u][0] = s[u][1] = s[u][2] = s[u][3] = 0.f;
      s2[u][0] = s2[u][1] = s2[u][2] = s2[u][3] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mma_16816(s[u], q[j].x, 0u, q[j].y, 0u, f.k[u][j].x, f.k[u][j].y);
        mma_16816(s2[u], q[j].z, 0u, q[j].w, 0u, f.k[u][j].z, f.k[u][j].w);
      }
#pragma unroll
    for (int u = 0; u < 2; ++u) { s[u][0] += s2[u][0]; s[u][1] += s2[u][1]; }
    if (next < n_tiles) load_k(next);                          // into the registers the first MMA has read
    if constexpr (kAhead) prefetch_tile<D>(kc, vc, pitch, pos, next + n_units);
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
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);             // the four lanes of a head: now the head's sum in each
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
}

}  // namespace attn
}  // namespace smr
