// One decode step (1 to 16 sequences) through up to eight decoder layers as ONE persistent kernel, for ranks with nobody
// to reduce with.  No upstream counterpart (the upstream recipes stop at the single fused op).
//
// What bounds it: the weights of a layer cross HBM once (214 MB for a TP8 share of the 70B layer, 30 us at the 7.1
// TB/s a pure TMA stream reaches); everything else is latency.  As five kernels that start under one another the
// same step took 60 us a layer: at every boundary an SM had nothing in flight from the last byte of one kernel
// (drain, epilogue, exit) to the first byte of the next (launch, set-up, first load).  Here
//   * one CTA per SM stays for the whole step, and its producer warp streams the weights of all phases of all layers
//     through one ring without ever waiting for activations: while the CTAs meet at a phase boundary, 150 KB per
//     SM (about 3 us of HBM) keep arriving;
//   * when they wait longer, DRAM goes on filling L2 with the weights that come next (see kAhead);
//   * a phase is a GEMM with the weight rows as the MMA's M and the batch (padded to 16) as its N; its rows are dealt
//     out evenly over the CTAs (tile i starts at floor(i N / tiles), so 8192 rows are 148 tiles of 55 or 56), K is
//     only split where a phase has too few rows (QKV), and then the attention adds the fp32 parts up;
//   * a CTA keeps its columns of the residual stream in shared memory; SiLU(gate) * up, the residual adds and the norms
//     happen on the way out, so that x comes in by TMA as it is;
//   * between phases the CTAs meet at a counter in global memory (release add by one thread, acquire poll by one
//     thread, about 1.3 us); attention is dealt out over (sequence, KV head, split of the context), then the sums of
//     the splits over (sequence, query head).  A layer has eight such round trips over the whole grid: six counters,
//     and twice, before a norm, the exchange of the sums of squares.
// The CTAs wait for one another, so the launch is cooperative.  Every wait is bounded.
// Two layers of that share, against the five kernels: batch 1 at position 3000 133 -> 105 us, batch 16 at 6500 172 -> 139
// us.  Their weights and caches at the measured copy rate take 66 and 82.
// Of the 87000 cycles a layer takes at batch 1 (52 us) 55000 are the weights (QKV 8700, o 5000, gate / up 28000, down 13700, each
// with its first load of x), 12000 the attention and the sum of its splits, 17000 the meeting points, 3000 the residual and the norm.
//
// Arithmetic is that of the single ops but for one rounding: gate and up reach SiLU as fp32 accumulators, where separate ops
// round them to bf16 first.  Else bf16 activations between phases, fp32 accumulation, the norm rounded before and after
// its weight, a projection rounded before its residual add, every sum in a fixed order.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../device/mbarrier.cuh"
#include "../device/tcgen05.cuh"
#include "../device/tma.cuh"
#include "../device/vec.cuh"
#include "../symm/driver_api.h"
#include "decode_attention.cuh"
#include "decode_stack.h"
#include "launch.h"
#include "residency.h"

namespace smr {

namespace {

constexpr int kMaxLayers = 8;                                   // per launch (kernel parameters)
constexpr int kBatchN = 16;                                     // MMA N: the batch, rows beyond it are zero
constexpr int kBK = 64;                                         // k per block = one 128-byte swizzle row
// warp 0: weights, warp 1: MMA, warps 2..7: the rest.  Eight warps, because a ninth would cut the registers per thread
// from 255 to 168, and the attention's spills then cost more than two more warps bring.
constexpr int kThreads = 256;
constexpr int kComputeWarp0 = 2, kWarps = 6, kCompute = kWarps * 32;
constexpr uint32_t kSlotBytes = 28672;                          // four k blocks of 56 rows, or two of 112
constexpr int kSlots = 6;
// The weight stream of an SM at a meeting point: a slot that has not become free for twice the time its bytes take at the
// SM's share of HBM (25 bytes a cycle) means that the phase is waiting, and then the steps after the ring go into
// L2 at that rate, up to six of them (25 MB over all SMs).  Two layers at batch 1 / batch 16: without 112.5 / 148.6, up
// to 4 steps 106.1 / 144.8, 6 104.7 / 145.0, 12 106.3 / 148.5 us; all the time instead of only when idle costs 7 us with
// 4 steps and 33 with 16.  Weights are loaded as the first to leave L2 (5 to 8 us slower before that): what stays
// are the activations, the new keys and values and what was prefetched.
constexpr int kAhead = 6;
constexpr int kShareOfHbm = 25, kIdleCycles = 2 * (int)kSlotBytes / kShareOfHbm;
constexpr int kGroupBlocks = 4;                                 // k blocks of x under one barrier
constexpr int kXGroups = 4;
constexpr uint32_t kXBlockBytes = kBatchN * kBK * 2;            // 2 KB
constexpr uint32_t kXOffset = kSlots * kSlotBytes;
// a phase's accumulator ([16][128] fp32), or the warps' attention results ([4][8][D + 4] fp32)
constexpr uint32_t kWorkOffset = kXOffset + kXGroups * kGroupBlocks * kXBlockBytes;
constexpr uint32_t kWorkBytes = 17408;
constexpr uint32_t kResidOffset = kWorkOffset + kWorkBytes;     // this CTA's columns of the residual stream [16][128] bf16
constexpr uint32_t kBarOffset = kResidOffset + 16 * 128 * 2;
constexpr uint32_t kNumBars = 2 * kSlots + 2 * kXGroups + 1;
constexpr uint32_t kSsOffset = kBarOffset + ((8 * kNumBars + 127) & ~127u);   // [12][16] fp32, then [16] scales
constexpr uint32_t kMlOffset = kSsOffset + 17 * 16 * 4;                       // attention: (max, sum) [6 warps][8 heads]
constexpr uint32_t kAngleOffset = kMlOffset + 8 * 8 * 8;                      // (cos, sin) [64]
constexpr uint32_t kRowOffset = kAngleOffset + 64 * 8;                        // attention: queries, key, value [10][D] bf16
constexpr uint32_t kMiscOffset = kRowOffset + 10 * 128 * 2;
constexpr uint32_t kSmemTotal = kMiscOffset + 32 + 1024;
constexpr int kMaxSplit = 64;
constexpr uint32_t kTmemCols = 32;
static_assert(kCompute == 192 && 16 * 128 * 4 <= kWorkBytes && 4 * 8 * 132 * 4 <= kWorkBytes, "work area");
static_assert(kSmemTotal <= 232448, "shared memory limit exceeded");

// Counters at which a layer's CTAs meet: what is complete there.  Before kNormedX1 and kNormedY they have met once more,
// at the sums of squares (`ss`).
enum Meet { kQkvDone = 0, kSplitsDone, kAttnDone, kNormedX1, kActDone, kNormedY, kMeets };
enum Phase { kQkv = 0, kO = 1, kGateUp = 2, kDown = 3 };

// How a phase's weight [N, K] is dealt out over the CTAs.
struct PhasePlan {
  int K, cols;            // k; output columns (rows of the weight, or of one half of it)
  int halves;             // 2: gate and up rows make one output column
  int tiles, ksplit;      // CTA i takes tile i / ksplit, part i % ksplit of K
  int box;                // columns a tile loads (the widest one's)
  int kb_per;             // k blocks per part
  int slot_blocks;        // k blocks in a ring slot: 1, 2 or 4, a divisor of every part's k blocks
  uint32_t block_bytes;   // distance of the k blocks in a slot (1024-byte multiple)
};

struct LayerParams {
  CUtensorMap w[4];
  const __nv_bfloat16 *norm1, *norm2;
  __nv_bfloat16 *k_cache, *v_cache;
};

struct StackParams {
  PhasePlan plan[4];
  int n_layers, batch, H, hq, hkv, D, s_max, n_split;
  int pos0;
  const int* pos_dev;
  float eps, scale, log2_theta;
  // activations and meeting points in global memory (scratch)
  const __nv_bfloat16* x;      // [batch, H] input of the first layer
  __nv_bfloat16* y;            // [batch, H] output of the last layer
  __nv_bfloat16* xn;           // [batch, H] the residual stream, normalised: operand of QKV and gate / up
  uint64_t* ss;                // [G][16] (sum of squares of a CTA's columns of the residual stream, which one: 1, 2, ...)
  float* qkv;                  // [ksplit][batch][(hq + 2 hkv) D] fp32 parts
  __nv_bfloat16* attn;         // [batch, hq D]
  __nv_bfloat16* act;          // [batch, F]
  float* partials;             // attention: [batch hkv][n_split][8][D + 4]
  uint32_t* meet;              // [n_layers][kMeets] arrivals; like `ss` zeroed by the kernel before this one
  uint64_t timeout_ns;
  Status* status;
  CUtensorMap x_map[4];        // the phases' activations: xn, attn, xn, act
  LayerParams layer[kMaxLayers];
};

__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 192;" ::: "memory"); }
__device__ __forceinline__ float round_bf16(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

// This CTA's part of a phase.
struct Share {
  bool any;               // false: no tile for this CTA
  int n0, n1;             // output columns
  int part;               // of K
  int kb0, n_kb;          // k blocks
  int n_steps;            // ring slots
};
__device__ __forceinline__ Share share_of(const PhasePlan& p, int cta) {
  Share s;
  const int tile = cta / p.ksplit;
  s.part = cta - tile * p.ksplit;
  s.any = tile < p.tiles;
  s.n0 = (int)((long long)tile * p.cols / p.tiles);
  s.n1 = (int)((long long)(tile + 1) * p.cols / p.tiles);
  const int kb_total = p.K / kBK;
  s.kb0 = s.part * p.kb_per;
  s.n_kb = (s.kb0 + p.kb_per < kb_total ? s.kb0 + p.kb_per : kb_total) - s.kb0;
  if (!s.any || s.n_kb < 0) s.n_kb = 0;
  s.n_steps = s.n_kb / p.slot_blocks;
  return s;
}

// Waits until every CTA has arrived at `counter` (their stores are visible afterwards).  All compute threads.
__device__ __forceinline__ bool await(uint8_t* smem, int ct, const uint32_t* counter, int n_ctas, uint64_t timeout_ns, Status* status) {
  int* flags = reinterpret_cast<int*>(smem + kMiscOffset + 8);
  if (ct == 0 && flags[0]) {
    if (!wait_ge_acquire_gpu(counter, (uint32_t)n_ctas, timeout_ns)) {
      report_status(status, kTimeoutFlag, 0, blockIdx.x, 0, kWhereGemvArrive);
      flags[0] = 0;
    }
  }
  compute_sync();
  return flags[0] != 0;
}

// x of a phase (k blocks [kb0, kb0 + n_kb)) into the MMA's B operand.  One thread.  `meet`: the counter that says x is
// complete, or nullptr.  `gx`: x groups this CTA has loaded so far.  Rows beyond the batch keep what the ring held:
// they only reach columns of D that nobody reads.
__device__ __forceinline__ bool load_x(uint8_t* smem, const CUtensorMap* map, const Share& sh, int batch, const uint32_t* meet,
                                       int n_ctas, uint32_t gx, uint64_t timeout_ns, Status* status) {
  uint64_t* x_full = reinterpret_cast<uint64_t*>(smem + kBarOffset) + 2 * kSlots;
  uint64_t* x_empty = x_full + kXGroups;
  if (meet != nullptr) {
    if (!wait_ge_acquire_gpu(meet, (uint32_t)n_ctas, timeout_ns)) {
      report_status(status, kTimeoutFlag, 0, blockIdx.x, 0, kWhereGemvArrive);
      return false;
    }
    asm volatile("fence.proxy.async.global;" ::: "memory");        // written by ordinary stores, read by TMA
  }
  for (int kb = 0; kb < sh.n_kb; kb += kGroupBlocks, ++gx) {
    const int slot = (int)(gx % kXGroups), n = sh.n_kb - kb < kGroupBlocks ? sh.n_kb - kb : kGroupBlocks;
    const uint32_t use = gx / kXGroups;
    if (use > 0 && !mbar_wait(&x_empty[slot], (use - 1) & 1u, timeout_ns)) {
      report_status(status, kTimeoutMbarrier, 0, blockIdx.x, slot, kWhereGemmEmpty);
      return false;
    }
    mbar_arrive_expect_tx(&x_full[slot], (uint32_t)(n * batch) * 128u);
    for (int j = 0; j < n; ++j)
      tma_load_2d(smem + kXOffset + (size_t)(slot * kGroupBlocks + j) * kXBlockBytes, map, &x_full[slot],
                  (sh.kb0 + kb + j) * kBK, 0);
  }
  return true;
}

// One (sequence, KV head, split) of the attention of layer `l`; `first`: the queries may not be there yet.
template <int D>
__device__ __forceinline__ bool attend_item(const StackParams& p, uint8_t* smem, int l, int item, int pos, bool first) {
  const int ct = (int)threadIdx.x - 32 * kComputeWarp0, cw = ct >> 5, lane = ct & 31;
  float* work = reinterpret_cast<float*>(smem + kWorkOffset);
  const float2* angles = reinterpret_cast<const float2*>(smem + kAngleOffset);
  float2* ml = reinterpret_cast<float2*>(smem + kMlOffset);        // [6 warps][8 heads] (max, sum)
  const int G = p.hq / p.hkv, bh_total = p.batch * p.hkv, n_qkv = (p.hq + 2 * p.hkv) * D;
  const int bh = item % bh_total, split = item / bh_total, b = bh / p.hkv, kvh = bh - b * p.hkv;
  const LayerParams& L = p.layer[l];
  const size_t base = ((size_t)b * p.s_max * p.hkv + kvh) * D;
  __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(smem + kRowOffset);   // [G queries, key, value][D]
  bool ok = true;
  const int unit = cw * p.n_split + split, n_units = p.n_split * kWarps, pitch = p.hkv * D;
  auto ready = [&] {                                               // this warp's first keys and values are on their way
    if (first) ok = await(smem, ct, p.meet + l * kMeets + kQkvDone, (int)gridDim.x, p.timeout_ns, p.status);
    // The new token's queries, key and value: the projection's K parts are added up here (all of them in flight at
    // once), rounded as a projection is, rotated as the stand-alone RoPE kernel rotates.  Four pairs (i, i + D / 2)
    // per thread.
    {
      const int parts = p.plan[kQkv].ksplit;
      const size_t part_stride = (size_t)p.batch * n_qkv;
      for (int i = ct; i < (G + 2) * D / 8; i += kCompute) {
        const int r = i / (D / 8), d = (i - r * (D / 8)) * 4;
        const int h = r < G ? kvh * G + r : (r == G ? p.hq + kvh : p.hq + p.hkv + kvh);
        const float* src = p.qkv + (size_t)b * n_qkv + (size_t)h * D + d;
        float4 v[2][8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < parts) {
            v[0][q] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)q * part_stride));
            v[1][q] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)q * part_stride + D / 2));
          }
        float x[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (q < parts) { a.x += v[half][q].x; a.y += v[half][q].y; a.z += v[half][q].z; a.w += v[half][q].w; }
          x[half][0] = round_bf16(a.x); x[half][1] = round_bf16(a.y);
          x[half][2] = round_bf16(a.z); x[half][3] = round_bf16(a.w);
        }
        if (r <= G) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 c = angles[d + e];
            const float lo = x[0][e], hi = x[1][e];
            x[0][e] = lo * c.x - hi * c.y;
            x[1][e] = hi * c.x + lo * c.y;
          }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
          *reinterpret_cast<uint2*>(row + r * D + half * (D / 2) + d) =
              make_uint2(pack_bf16x2(x[half][0], x[half][1]), pack_bf16x2(x[half][2], x[half][3]));
      }
      compute_sync();
    }
  };
  attn::State<D> st;
  attn::attend<D, true>(L.k_cache + base, L.v_cache + base, (size_t)pitch, pos, unit, n_units, G, p.scale, nullptr, ready,
                  [&](int part, int head, int d) {
                    const int r = part == 0 ? head : G + part - 1;
                    return *reinterpret_cast<const Vec16*>(row + r * D + d);
                  },
                  st);
  if (!ok) return false;
  const int g = lane >> 2, t = lane & 3;
  // ---- the six warps: 4 and 5 leave their results, 0 and 1 add theirs, 2 and 3 leave theirs: four in `work` ----
  // Dimensions 64 i + 8 g + 4 c .. + 3 of a head as one 16-byte access; rows of D + 4 floats, so that the four heads of a
  // quarter warp fall into different banks (8-way conflicts and scalar stores before: 1.4 us for the merge).
  constexpr int kPitch = D + 4;
  auto slot_of = [&](int w, int head, int i, int c) {
    return reinterpret_cast<float4*>(work + ((size_t)w * 8 + head) * kPitch + i * 64 + g * 8 + 4 * c);
  };
  auto mine_of = [&](int u, int i, int c) {                        // of head 2t + u
    return make_float4(st.acc[i * 4 + 2 * c][u], st.acc[i * 4 + 2 * c][u + 2], st.acc[i * 4 + 2 * c + 1][u],
                       st.acc[i * 4 + 2 * c + 1][u + 2]);
  };
  if (t == 0) ml[cw * 8 + g] = make_float2(st.m, st.l);
  if (cw >= 2) {
    const int to = cw >= 4 ? cw - 4 : cw;
#pragma unroll
    for (int i = 0; i < D / 64; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) *slot_of(to, 2 * t + (c & 1), i, c >> 1) = mine_of(c & 1, i, c >> 1);
  }
  compute_sync();
  if (cw < 2) {
    float f0[2], f1[2];                                            // weights of this warp's and of the other's result
#pragma unroll
    for (int u = 0; u < 2; ++u) {                                  // heads 2t and 2t + 1
      const float m0 = ml[cw * 8 + 2 * t + u].x, m1 = ml[(cw + 4) * 8 + 2 * t + u].x, big = fmaxf(m0, m1);
      f0[u] = exp2f(m0 - big);
      f1[u] = exp2f(m1 - big);
    }
#pragma unroll
    for (int i = 0; i < D / 64; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int u = c & 1;
        float4* s = slot_of(cw, 2 * t + u, i, c >> 1);
        const float4 mv = mine_of(u, i, c >> 1), ov = *s;
        *s = make_float4(f0[u] * mv.x + f1[u] * ov.x, f0[u] * mv.y + f1[u] * ov.y, f0[u] * mv.z + f1[u] * ov.z,
                         f0[u] * mv.w + f1[u] * ov.w);
      }
    __syncwarp();
    if (t == 0) {                                                  // head g of this pair of warps
      const float2 a = ml[cw * 8 + g], c = ml[(cw + 4) * 8 + g];
      const float big = fmaxf(a.x, c.x);
      ml[cw * 8 + g] = make_float2(big, exp2f(a.x - big) * a.y + exp2f(c.x - big) * c.y);
    }
  }
  compute_sync();
  // ---- a warp per head, D / 32 dimensions per lane ----
  constexpr int kVec = D / 32, kRec = D + 4;                   // a record: D weighted-V sums, max, sum (and two unused)
  using VecT = typename std::conditional<kVec == 4, float4, float2>::type;
  auto add_scaled = [](VecT& a, float f, const VecT& v) {
    a.x += f * v.x; a.y += f * v.y;
    if constexpr (kVec == 4) { a.z += f * v.z; a.w += f * v.w; }
  };
  float* mine = p.partials + ((size_t)bh * p.n_split + split) * 8 * kRec;
  __nv_bfloat16* out = p.attn + ((size_t)b * p.hq + (size_t)kvh * G) * D;
  auto store_out = [&](int h, const VecT& a, float sum) {
    const float inv = 1.0f / sum;
    __nv_bfloat16* o = out + (size_t)h * D + lane * kVec;
    if constexpr (kVec == 4)
      *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(a.x * inv, a.y * inv), pack_bf16x2(a.z * inv, a.w * inv));
    else
      *reinterpret_cast<uint32_t*>(o) = pack_bf16x2(a.x * inv, a.y * inv);
  };
  for (int h = cw; h < G; h += kWarps) {
    float big = attn::kNoScore, sum = 0.f;
    VecT a{};
    float2 r[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      r[w] = ml[w * 8 + h];
      big = fmaxf(big, r[w].x);
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = exp2f(r[w].x - big);
      sum += f * r[w].y;
      add_scaled(a, f, *reinterpret_cast<const VecT*>(work + ((size_t)w * 8 + h) * kPitch + lane * kVec));
    }
    if (p.n_split == 1) {
      store_out(h, a, sum);
    } else {
      *reinterpret_cast<VecT*>(mine + h * kRec + lane * kVec) = a;
      if (lane == 0) *reinterpret_cast<float2*>(mine + h * kRec + D) = make_float2(big, sum);
    }
  }
  compute_sync();                                                  // `work` may be reused
  return true;
}

// The splits of the attention of (sequence, query head) `item` added up: warp w takes splits w, w + 6, ..., all their
// records in flight at once.
template <int D>
__device__ __forceinline__ void combine_item(const StackParams& p, uint8_t* smem, int item) {
  constexpr int kVec = D / 32, kRec = D + 4, kMine = (kMaxSplit + kWarps - 1) / kWarps;
  using VecT = typename std::conditional<kVec == 4, float4, float2>::type;
  const int ct = (int)threadIdx.x - 32 * kComputeWarp0, cw = ct >> 5, lane = ct & 31;
  float* work = reinterpret_cast<float*>(smem + kWorkOffset);      // [6][D] sums, then the six totals
  const int G = p.hq / p.hkv, b = item / p.hq, h = item - b * p.hq, bh = b * p.hkv + h / G;
  const float* all = p.partials + ((size_t)bh * p.n_split * 8 + h % G) * kRec;
  VecT v[kMine];
  float2 ml[2];
#pragma unroll
  for (int u = 0; u < kMine; ++u) {
    const int i = cw + kWarps * u;
    if (i < p.n_split) v[u] = __ldcg(reinterpret_cast<const VecT*>(all + (size_t)i * 8 * kRec + lane * kVec));
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = lane + 32 * u;
    ml[u] = i < p.n_split ? __ldcg(reinterpret_cast<const float2*>(all + (size_t)i * 8 * kRec + D))
                          : make_float2(attn::kNoScore, 0.f);
  }
  float big = fmaxf(ml[0].x, ml[1].x), total = 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
  float w[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    w[u] = lane + 32 * u < p.n_split ? exp2f(ml[u].x - big) : 0.f;  // 0 for a split that saw no position
    total += w[u] * ml[u].y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  VecT a{};
#pragma unroll
  for (int u = 0; u < kMine; ++u) {
    const int i = cw + kWarps * u;
    const float f = __shfl_sync(0xffffffffu, i < 32 ? w[0] : w[1], i & 31);
    if (i < p.n_split) {
      a.x += f * v[u].x; a.y += f * v[u].y;
      if constexpr (kVec == 4) { a.z += f * v[u].z; a.w += f * v[u].w; }
    }
  }
  *reinterpret_cast<VecT*>(work + cw * D + lane * kVec) = a;
  compute_sync();
  const float inv = 1.0f / total;                                  // the same in every warp
  for (int d = ct * 2; d < D; d += 2 * kCompute) {
    float x = 0.f, y = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const float2 r = *reinterpret_cast<const float2*>(work + i * D + d);
      x += r.x; y += r.y;
    }
    *reinterpret_cast<uint32_t*>(p.attn + (size_t)item * D + d) = pack_bf16x2(x * inv, y * inv);
  }
  compute_sync();                                                  // `work` may be reused
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) decode_stack_kernel(const __grid_constant__ StackParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBarOffset);
  uint64_t* w_full = bars;
  uint64_t* w_empty = bars + kSlots;
  uint64_t* x_full = bars + 2 * kSlots;
  uint64_t* x_empty = bars + 2 * kSlots + kXGroups;
  uint64_t* tmem_full = bars + 2 * kSlots + 2 * kXGroups;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kMiscOffset);
  int* flags = reinterpret_cast<int*>(smem + kMiscOffset + 8);     // [0] all waits fine
  float* work = reinterpret_cast<float*>(smem + kWorkOffset);
  __nv_bfloat16* resid = reinterpret_cast<__nv_bfloat16*>(smem + kResidOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = (int)blockIdx.x, n_ctas = (int)gridDim.x;
  bool failed = false;

  if (threadIdx.x == 0) {
    for (int i = 0; i < (int)kNumBars; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
    flags[0] = 1;
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish_alloc_permit();
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  tcgen05_fence_after_thread_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- the weight stream of the whole step ----------------
    if (elect_one()) {
      // Ring slot `i` of phase `step` (of layer step / 4): a cursor over all the loads of this CTA.
      struct Cursor {
        int step, i;
        Share sh;
      };
      const int n_phases = 4 * p.n_layers;
      auto settle = [&](Cursor& c) {                               // on a step that exists, or at the end
        while (c.i >= c.sh.n_steps && ++c.step < n_phases) {
          c.i = 0;
          c.sh = share_of(p.plan[c.step & 3], cta);
        }
      };
      Cursor at{0, 0, share_of(p.plan[0], cta)}, ahead = at;
      settle(at);
      int slot = 0, lead = 0;                                      // lead: steps from `at` to `ahead`, in L2 or on their way there
      uint32_t use = 0;                                            // times the ring has wrapped
      while (at.step < n_phases) {
        const PhasePlan& pl = p.plan[at.step & 3];
        if (use > 0) {
          Deadline d(p.timeout_ns);
          const long long t0 = clock64();
          long long due = kIdleCycles;
          while (!mbar_test(&w_empty[slot], (use - 1) & 1u)) {
            if (lead < kAhead && ahead.step < n_phases && clock64() - t0 >= due) {
              const PhasePlan& next = p.plan[ahead.step & 3];
              for (int j = 0; j < next.slot_blocks; ++j)
                tma_prefetch_4d(&p.layer[ahead.step >> 2].w[ahead.step & 3], 0, ahead.sh.n0, 0,
                                ahead.sh.kb0 + ahead.i * next.slot_blocks + j);
              due += next.slot_blocks * next.box * next.halves * 128 / kShareOfHbm;
              ++ahead.i;
              settle(ahead);
              ++lead;
            }
            if (!d.alive()) {
              report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, slot, kWhereGemmEmpty, at.step);
              failed = true;
              break;
            }
          }
          if (failed) break;
        }
        mbar_arrive_expect_tx(&w_full[slot], (uint32_t)(pl.box * pl.halves) * 128u * (uint32_t)pl.slot_blocks);
        for (int j = 0; j < pl.slot_blocks; ++j)
          tma_load_4d_once(smem + (size_t)slot * kSlotBytes + (size_t)j * pl.block_bytes,
                           &p.layer[at.step >> 2].w[at.step & 3], &w_full[slot], 0, at.sh.n0, 0,
                           at.sh.kb0 + at.i * pl.slot_blocks + j);
        if (++slot == kSlots) { slot = 0; ++use; }
        ++at.i;
        settle(at);
        if (lead > 0) --lead;
        else ahead = at;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issue ----------------
    // The issuing thread must not need more than 250 cycles per k block of a full-width phase.  Measured on a loop
    // of this shape (M 64): 92 cycles for the four MMAs alone, 250 with a wait, a commit and a run-time number of
    // blocks per slot, 155 with the number fixed at two and the next slot's barrier tested before this slot's
    // MMAs go out.  A wait that runs out is remembered and not acted upon, to keep the loop free of exits.
    if (elect_one()) {
      int slot = 0, xs = 0;
      uint32_t wphase = 0, xphase = 0;
      auto run = [&](auto blocks, const PhasePlan& pl, const Share& sh) {
        constexpr int NB = decltype(blocks)::value;
        const uint32_t idesc = umma_idesc_bf16_f32(pl.box * pl.halves <= 64 ? 64 : 128, kBatchN);
        bool w_ready = false, x_ready = false;
        for (int i = 0; i < sh.n_steps; ++i) {
          const int kb = i * NB;
          if ((kb & (kGroupBlocks - 1)) == 0 && !x_ready) failed |= !mbar_wait(&x_full[xs], xphase, failed ? 0 : p.timeout_ns);
          if (!w_ready) failed |= !mbar_wait(&w_full[slot], wphase, failed ? 0 : p.timeout_ns);
          tcgen05_fence_after_thread_sync();
          const bool group_ends = ((kb + NB) & (kGroupBlocks - 1)) == 0 || i == sh.n_steps - 1;
          const int slot1 = slot + 1 == kSlots ? 0 : slot + 1, xs1 = xs + 1 == kXGroups ? 0 : xs + 1;
          w_ready = i + 1 < sh.n_steps && mbar_test(&w_full[slot1], wphase ^ (slot1 == 0 ? 1u : 0u));
          x_ready = group_ends && i + 1 < sh.n_steps && mbar_test(&x_full[xs1], xphase ^ (xs1 == 0 ? 1u : 0u));
          const uint32_t sw = smem_u32(smem) + (uint32_t)slot * kSlotBytes;
          const uint32_t sx = smem_u32(smem + kXOffset) + (uint32_t)(xs * kGroupBlocks + (kb & (kGroupBlocks - 1))) * kXBlockBytes;
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const uint64_t da = umma_smem_desc_sw128(sw + (uint32_t)j * pl.block_bytes);
            const uint64_t db = umma_smem_desc_sw128(sx + (uint32_t)j * kXBlockBytes);
#pragma unroll
            for (int k = 0; k < 4; ++k)                            // +16 k = +32 bytes of the 128-byte rows
              umma_bf16_ss(tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (i | j | k) != 0 ? 1u : 0u);
          }
          umma_commit(&w_empty[slot]);
          if (group_ends) {
            umma_commit(&x_empty[xs]);
            xs = xs1;
            if (xs1 == 0) xphase ^= 1;
          }
          slot = slot1;
          if (slot1 == 0) wphase ^= 1;
        }
        umma_commit(tmem_full);
      };
      for (int l = 0; l < p.n_layers; ++l) {
        for (int ph = 0; ph < 4; ++ph) {
          const PhasePlan& pl = p.plan[ph];
          const Share sh = share_of(pl, cta);
          if (sh.n_steps == 0) continue;
          if (pl.slot_blocks == 4) run(std::integral_constant<int, 4>{}, pl, sh);
          else if (pl.slot_blocks == 2) run(std::integral_constant<int, 2>{}, pl, sh);
          else run(std::integral_constant<int, 1>{}, pl, sh);
          if (failed) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, slot, kWhereGemmFull, l * 4 + ph);
        }
      }
    }
  } else {
    // ---------------- activations: staging, epilogues, attention, meeting points ----------------
    const int ct = (int)threadIdx.x - 32 * kComputeWarp0, cw = warp - kComputeWarp0;
    uint32_t gx = 0;                                               // x groups staged so far
    uint32_t acc_uses = 0;                                         // accumulators read so far
    // Meeting point `i`: every CTA has finished the phase (its stores are visible after `await`).
    auto arrive = [&](int i) {
      compute_sync();
      if (ct == 0) {
        red_add_release_gpu(p.meet + i, 1u);                       // releases what the barrier has ordered before it
      }
    };
    // The last compute warp (its TMEM lanes are nobody's) feeds x to the MMA; the others go on to the accumulator.
    auto stage = [&](int ph, const Share& sh, int meet) {
      if (warp == kComputeWarp0 + kWarps - 1 && sh.any) {
        if (lane == 0 && !load_x(smem, &p.x_map[ph], sh, p.batch, meet < 0 ? nullptr : p.meet + meet, n_ctas, gx, p.timeout_ns,
                                 p.status))
          flags[0] = 0;
        __syncwarp();
      }
      gx += (uint32_t)((sh.n_kb + kGroupBlocks - 1) / kGroupBlocks);
    };
    // The phase's accumulator into `work` [16][128] (row = row of the tile), visible to all compute threads.
    auto fetch_accumulator = [&](const PhasePlan& pl) -> bool {
      if (cw < 4) {
        if (!mbar_wait(tmem_full, acc_uses & 1u, p.timeout_ns)) {
          if (lane == 0) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, 0, kWhereGemmTmemFull);
          flags[0] = 0;
        } else {
          tcgen05_fence_after_thread_sync();
          const int quarter = warp & 3;
          uint32_t acc[16];
          tmem_ld_32x32b_x16(tmem + ((uint32_t)(quarter * 32) << 16), acc);
          tmem_ld_wait();
          tcgen05_fence_before_thread_sync();
          // an MMA of 64 rows leaves sixteen of them in each quarter of the lanes
          const bool m64 = pl.box * pl.halves <= 64;
          const int row = m64 ? quarter * 16 + lane : quarter * 32 + lane;
          if (!m64 || lane < 16) {
#pragma unroll
            for (int b = 0; b < 16; ++b)
              if (b < p.batch) work[b * 128 + row] = __uint_as_float(acc[b]);
          }
        }
      }
      ++acc_uses;
      compute_sync();
      return flags[0] != 0;
    };
    // Residual stream: resid = bf16(bf16(product) + resid) on this CTA's columns (the same ones after o and after down),
    // into `out` when that is given, else its sums of squares into ss[cta][b], marked `mark`.
    auto add_residual = [&](const PhasePlan& pl, const Share& sh, __nv_bfloat16* out, uint32_t mark) {
      const int width = sh.any ? sh.n1 - sh.n0 : 0;
      for (int b = cw; b < p.batch; b += kWarps) {
        float t = 0.f;
        for (int col = lane; col < width; col += 32) {
          const __nv_bfloat16 v = __float2bfloat16_rn(round_bf16(work[b * 128 + col]) + __bfloat162float(resid[b * 128 + col]));
          resid[b * 128 + col] = v;
          if (out != nullptr) out[(size_t)b * pl.cols + sh.n0 + col] = v;
          const float f = __bfloat162float(v);
          t += f * f;
        }
        if (out != nullptr) continue;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0)
          asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p.ss + (size_t)cta * 16 + b),
                       "l"((uint64_t)mark << 32 | __float_as_uint(t)) : "memory");
      }
    };
    // This CTA's columns of the residual stream, normalised: xn = bf16(bf16(x * scale) * w).  Done once per column and
    // not by every CTA for all of x: at batch 16 that took 6 warps 42000 cycles for gate / up, whose weights take
    // 29000 to arrive, against one more meeting point.  The sums carry the mark of their norm, so the wait for the
    // other CTAs and the read of their sums are the same load.
    auto normalise = [&](const Share& sh, const __nv_bfloat16* w, uint32_t mark) -> bool {
      float wv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int col = lane + 32 * c;
        wv[c] = sh.any && col < sh.n1 - sh.n0 ? __bfloat162float(w[sh.n0 + col]) : 0.f;
      }
      float* red = reinterpret_cast<float*>(smem + kSsOffset);     // [12][16], then the 16 scales
      const int rb = ct & 15, r = ct >> 4;
      float t = 0.f;
      if (rb < p.batch) {
        for (int i0 = r; i0 < n_ctas; i0 += 156) {                 // thirteen loads in flight: one round trip for 148 CTAs
          uint64_t v[13];
          Deadline d(p.timeout_ns);
          for (;;) {
            bool there = true;
#pragma unroll
            for (int u = 0; u < 13; ++u) {
              v[u] = (uint64_t)mark << 32;                         // + 0.0f
              if (i0 + 12 * u < n_ctas)
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[u]) : "l"(p.ss + (i0 + 12 * u) * 16 + rb) : "memory");
            }
#pragma unroll
            for (int u = 0; u < 13; ++u) there = there && (uint32_t)(v[u] >> 32) == mark;
            if (there) break;
            if (!d.alive()) {
              report_status(p.status, kTimeoutFlag, 0, blockIdx.x, 0, kWhereGemvArrive);
              flags[0] = 0;
              break;
            }
          }
#pragma unroll
          for (int u = 0; u < 13; ++u) t += __uint_as_float((uint32_t)v[u]);
        }
      }
      red[r * 16 + rb] = t;
      compute_sync();
      if (!flags[0]) return false;
      if (!sh.any) return true;
      if (ct < 16) {
        t = 0.f;
#pragma unroll
        for (int i = 0; i < 12; ++i) t += red[i * 16 + ct];
        red[12 * 16 + ct] = rsqrtf(t / (float)p.H + p.eps);
      }
      compute_sync();
      for (int b = cw; b < p.batch; b += kWarps) {
        const float scale = red[12 * 16 + b];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int col = lane + 32 * c;
          if (col < sh.n1 - sh.n0)
            p.xn[(size_t)b * p.H + sh.n0 + col] = __float2bfloat16_rn(round_bf16(__bfloat162float(resid[b * 128 + col]) * scale) * wv[c]);
        }
      }
      return true;
    };
    // The keys and values of this CTA's first share of the attention into L2, two tiles per warp, while the queries are still
    // being made (DRAM idles at the meeting points: the weight ring is full by then).
    auto prefetch_kv = [&](int l, int pos) {
      const int bh_total = p.batch * p.hkv, bh = cta % bh_total, split = cta / bh_total;
      if (split >= p.n_split) return;
      const int b = bh / p.hkv, kvh = bh - b * p.hkv, pitch = p.hkv * D, n_units = p.n_split * kWarps;
      const size_t base = ((size_t)b * p.s_max * p.hkv + kvh) * D;
      for (int i = 0, unit = cw * p.n_split + split; i < 2; ++i, unit += n_units)
        attn::prefetch_tile<D>(p.layer[l].k_cache + base, p.layer[l].v_cache + base, (size_t)pitch, pos, unit);
    };

    int pos = p.pos_dev != nullptr ? *p.pos_dev : p.pos0;
    pos = pos < 0 ? 0 : (pos >= p.s_max ? p.s_max - 1 : pos);
    float2* angles = reinterpret_cast<float2*>(smem + kAngleOffset);
    attn::fill_angles<D>(angles, ct, pos, p.log2_theta);           // read after the first compute_sync
    const int bh_total = p.batch * p.hkv, n_qkv = (p.hq + 2 * p.hkv) * D;

    const Share sh_x = share_of(p.plan[kO], cta);                  // columns of the residual stream
    if (sh_x.any)
      for (int b = cw; b < p.batch; b += kWarps)
        for (int col = lane; col < sh_x.n1 - sh_x.n0; col += 32) resid[b * 128 + col] = p.x[(size_t)b * p.H + sh_x.n0 + col];

    // One copy of the code for the four phases: at its first pass an SM fetches every instruction from L2 or beyond.
    bool ok = true;
#pragma unroll 1
    for (int step = 0; ok && step < 4 * p.n_layers; ++step) {
      const int l = step >> 2, ph = step & 3, meet = l * kMeets;
      const PhasePlan& pl = p.plan[ph];
      const Share sh = share_of(pl, cta);
      int x_done = meet + kActDone;
      if (ph == kQkv) {
        prefetch_kv(l, pos);
        x_done = l == 0 ? -1 : meet - kMeets + kNormedY;
      } else if (ph == kO) {
        x_done = meet + (p.n_split > 1 ? kAttnDone : kSplitsDone);
      } else if (ph == kGateUp) {
        x_done = meet + kNormedX1;
      }
      stage(ph, sh, x_done);
      if (sh.any) ok = fetch_accumulator(pl);
      if (!ok) break;
      const int width = sh.any ? sh.n1 - sh.n0 : 0;
      if (ph == kQkv) {  // fp32 parts, added up by the attention
        for (int b = cw; b < p.batch; b += kWarps)
          for (int c = lane; c < width; c += 32)
            p.qkv[((size_t)sh.part * p.batch + b) * n_qkv + sh.n0 + c] = work[b * 128 + c];
        arrive(meet + kQkvDone);
        for (int item = cta; ok && item < bh_total * p.n_split; item += n_ctas) ok = attend_item<D>(p, smem, l, item, pos, item == cta);
        arrive(meet + kSplitsDone);
        if (ok && p.n_split > 1) {
          if (cta < p.batch * p.hq) ok = await(smem, ct, p.meet + meet + kSplitsDone, n_ctas, p.timeout_ns, p.status);
          for (int item = cta; ok && item < p.batch * p.hq; item += n_ctas) combine_item<D>(p, smem, item);
          arrive(meet + kAttnDone);
        }
      } else if (ph == kGateUp) {  // SiLU(gate) * up
        for (int b = cw; b < p.batch; b += kWarps)
          for (int c = lane; c < width; c += 32) {
            const float g = work[b * 128 + c], u = work[b * 128 + pl.box + c];
            p.act[(size_t)b * pl.cols + sh.n0 + c] = __float2bfloat16_rn(g / (1.0f + __expf(-g)) * u);
          }
        arrive(meet + kActDone);
      } else {  // residual add, then the norm of the next projection
        const bool end = ph == kDown && l == p.n_layers - 1;
        const uint32_t mark = (uint32_t)(2 * l + (ph == kDown) + 1);
        add_residual(pl, sh, end ? p.y : nullptr, mark);
        if (!end) {
          ok = normalise(sh, ph == kO ? p.layer[l].norm2 : p.layer[l + 1].norm1, mark);
          arrive(meet + (ph == kO ? kNormedX1 : kNormedY));
        }
      }
    }
    failed = !ok;
  }

  if (__any_sync(0xffffffffu, failed)) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);               // let the loads in flight land
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  tcgen05_fence_after_thread_sync();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// The input's rows normalised for the first layer (one CTA per row), and the meeting points of the step back to zero.
// Everything is loaded up front: one trip to memory.
__global__ void __launch_bounds__(512)
decode_head_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ xn, int H,
                   float eps, uint4* meets, int n_meets) {
  constexpr int kKept = 4;                                         // 16-byte pieces of a row a thread keeps: H <= 16384
  const Vec16* xr = reinterpret_cast<const Vec16*>(x + (size_t)blockIdx.x * H);
  const Vec16* wr = reinterpret_cast<const Vec16*>(w);
  const int n = H / 8;
  Vec16 xv[kKept], wv[kKept];
#pragma unroll
  for (int u = 0; u < kKept; ++u) {
    const int i = (int)threadIdx.x + 512 * u;
    xv[u] = wv[u] = Vec16{0u, 0u, 0u, 0u};
    if (i < n) { xv[u] = ld_16_nc(xr + i); wv[u] = ld_16_nc(wr + i); }
  }
  for (int i = blockIdx.x * 512 + threadIdx.x; i < n_meets; i += gridDim.x * 512) meets[i] = make_uint4(0u, 0u, 0u, 0u);
  float t = 0.f;
  auto add = [&](const Vec16& v) {
    const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) t += bf16lo_to_f32(e[q]) * bf16lo_to_f32(e[q]) + bf16hi_to_f32(e[q]) * bf16hi_to_f32(e[q]);
  };
#pragma unroll
  for (int u = 0; u < kKept; ++u) add(xv[u]);
  for (int i = (int)threadIdx.x + 512 * kKept; i < n; i += 512) add(ld_16_nc(xr + i));
  __shared__ float warp_sums[16];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = t;
  __syncthreads();
  t = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) t += warp_sums[i];
  const float s = rsqrtf(t / (float)H + eps);
  auto two = [s](uint32_t a, uint32_t g) {
    return pack_bf16x2(round_bf16(bf16lo_to_f32(a) * s) * bf16lo_to_f32(g), round_bf16(bf16hi_to_f32(a) * s) * bf16hi_to_f32(g));
  };
  auto put = [&](int i, const Vec16& v, const Vec16& g) {
    *reinterpret_cast<uint4*>(xn + (size_t)blockIdx.x * H + (size_t)i * 8) =
        make_uint4(two(v.x, g.x), two(v.y, g.y), two(v.z, g.z), two(v.w, g.w));
  };
#pragma unroll
  for (int u = 0; u < kKept; ++u) {
    const int i = (int)threadIdx.x + 512 * u;
    if (i < n) put(i, xv[u], wv[u]);
  }
  for (int i = (int)threadIdx.x + 512 * kKept; i < n; i += 512) put(i, ld_16_nc(xr + i), ld_16_nc(wr + i));
}

// Rows of a weight [N, K] (or of its two halves) over `ctas` CTAs: one tile each and no split of K where that gives
// tiles worth an MMA, else K split in 2, 4 or 8.  A k block costs a CTA its bytes at the SM's share of HBM (25
// bytes a cycle) and at least 130 cycles of MMA and barrier work.
int plan_phase(int N, int K, int halves, bool may_split, int ctas, PhasePlan& out) {
  const int cols = N / halves, most = 128 / halves;
  double best = -1;
  for (int ks = 1; ks <= (may_split ? 8 : 1); ks *= 2) {
    const int kb_total = K / kBK;
    if (ks > 1 && kb_total < 4 * ks) break;
    int tiles = ctas / ks;
    if (tiles < 1) break;
    if (tiles > cols) tiles = cols;
    const int box = (cols + tiles - 1) / tiles;
    if (box > most) continue;
    // parts in whole groups of x, so that a part starts at a group
    int kb_per = (kb_total + ks - 1) / ks;
    if (ks > 1) kb_per = (kb_per + kGroupBlocks - 1) / kGroupBlocks * kGroupBlocks;
    if ((ks - 1) * kb_per >= kb_total) continue;                   // no part may be empty
    const double bytes = (double)box * halves * 128.0 / 25.0;
    const double cost = kb_per * (bytes > 130 ? bytes : 130.0);
    if (best >= 0 && cost > 0.95 * best) continue;
    best = cost;
    out.K = K; out.cols = cols; out.halves = halves;
    out.tiles = tiles; out.ksplit = ks; out.box = box; out.kb_per = kb_per;
    const int bytes1 = (box * halves * 128 + 1023) / 1024 * 1024;
    out.block_bytes = (uint32_t)bytes1;
    int nb = 4;
    while (nb > 1 && (bytes1 * nb > (int)kSlotBytes || kb_total % nb != 0 || kb_per % nb != 0)) nb >>= 1;
    out.slot_blocks = nb;
  }
  return best < 0 ? 1 : 0;
}

struct Layout {
  size_t xn, qkv, attn, act, y[2], partials, ss, meet, total;     // ss and meet side by side, zeroed together
  int n_split;
};

int make_plan(int batch, int H, int F, int hq, int hkv, int D, int s_max, int ctas, PhasePlan (&plan)[4], Layout& lo) {
  if (batch < 1 || batch > kBatchN || (D != 64 && D != 128) || hkv < 1 || hq % hkv != 0 || hq / hkv > attn::kHeads ||
      H % kBK != 0 || F % kBK != 0 || (hq * D) % kBK != 0 || H < kBK || F < kBK || s_max < 1 || ctas < 1)
    return 1;
  const int n_qkv = (hq + 2 * hkv) * D;
  if (plan_phase(n_qkv, H, 1, true, ctas, plan[kQkv]) || plan_phase(H, hq * D, 1, false, ctas, plan[kO]) ||
      plan_phase(2 * F, H, 2, false, ctas, plan[kGateUp]) || plan_phase(H, F, 1, false, ctas, plan[kDown]))
    return 1;
  const int rows = batch * hkv;
  int n = ctas / rows;
  const int by_length = (s_max + attn::kTile * kWarps - 1) / (attn::kTile * kWarps);
  if (n > by_length) n = by_length;
  lo.n_split = n < 1 ? 1 : (n > kMaxSplit ? kMaxSplit : n);
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~(size_t)255; return o; };
  lo.xn = take((size_t)batch * H * 2);
  lo.qkv = take((size_t)plan[kQkv].ksplit * batch * n_qkv * 4);
  lo.attn = take((size_t)batch * hq * D * 2);
  lo.act = take((size_t)batch * F * 2);
  for (int i = 0; i < 2; ++i) lo.y[i] = take((size_t)batch * H * 2);
  lo.partials = take((size_t)rows * lo.n_split * 8 * (D + 4) * 4);
  lo.ss = take((size_t)ctas * 16 * 8);
  lo.meet = take((size_t)kMaxLayers * kMeets * 4);
  lo.total = at;
  return 0;
}

// W [N, K] seen as [K / 64][halves][rows of a half][64 k]: a box is one k block of a tile, a complete K-major operand.
int encode_blocks(CUtensorMap* map, const void* base, const PhasePlan& pl) {
  const uint64_t K = (uint64_t)pl.K, rows = (uint64_t)pl.cols;
  cuuint64_t dims[4] = {(cuuint64_t)kBK, rows, (cuuint64_t)pl.halves, K / kBK};
  cuuint64_t strides[3] = {K * 2, rows * K * 2, (cuuint64_t)kBK * 2};
  cuuint32_t box[4] = {(cuuint32_t)kBK, (cuuint32_t)pl.box, (cuuint32_t)pl.halves, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = DriverApi::get().cuTensorMapEncodeTiled(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1;
}

// x [batch, K]: a box is one k block of all rows.
int encode_x(CUtensorMap* map, const void* base, int K, int batch) {
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)batch};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)batch};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = DriverApi::get().cuTensorMapEncodeTiled(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1;
}

template <int D>
int launch_steps(const DecodeStackArgs& a, const PhasePlan (&plan)[4], const Layout& lo, cudaStream_t stream) {
  auto kernel = decode_stack_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemTotal);
  if (e != cudaSuccess) return (int)e;
  if (int rc = check_co_resident(kernel, a.num_sms, kThreads, kSmemTotal)) return rc;
  char* s = static_cast<char*>(a.scratch);
  auto at = [&](size_t off) { return s + off; };
  for (int l0 = 0; l0 < a.n_layers; l0 += kMaxLayers) {
    const int n = a.n_layers - l0 < kMaxLayers ? a.n_layers - l0 : kMaxLayers;
    const bool last = l0 + n == a.n_layers;
    const void* x = l0 == 0 ? a.x : at(lo.y[1 - (l0 / kMaxLayers) % 2]);
    StackParams p{};
    for (int i = 0; i < 4; ++i) p.plan[i] = plan[i];
    p.n_layers = n;
    p.batch = a.batch; p.H = a.hidden; p.hq = a.hq; p.hkv = a.hkv; p.D = D; p.s_max = a.s_max;
    p.n_split = lo.n_split;
    p.pos0 = a.pos0;
    p.pos_dev = a.pos_dev;
    p.eps = a.eps;
    p.scale = 1.4426950408889634f / sqrtf((float)D);               // scores in units of log2
    p.log2_theta = log2f(a.rope_theta);
    p.x = static_cast<const __nv_bfloat16*>(x);
    p.y = static_cast<__nv_bfloat16*>(last ? a.y : static_cast<void*>(at(lo.y[(l0 / kMaxLayers) % 2])));
    p.xn = reinterpret_cast<__nv_bfloat16*>(at(lo.xn));
    p.ss = reinterpret_cast<uint64_t*>(at(lo.ss));
    p.qkv = reinterpret_cast<float*>(at(lo.qkv));
    p.attn = reinterpret_cast<__nv_bfloat16*>(at(lo.attn));
    p.act = reinterpret_cast<__nv_bfloat16*>(at(lo.act));
    p.partials = reinterpret_cast<float*>(at(lo.partials));
    p.meet = reinterpret_cast<uint32_t*>(at(lo.meet));
    p.timeout_ns = a.timeout_ns;
    p.status = a.status;
    const void* operand[4] = {p.xn, p.attn, p.xn, p.act};
    for (int i = 0; i < 4; ++i)
      if (encode_x(&p.x_map[i], operand[i], plan[i].K, a.batch)) return cudaErrorInvalidValue;
    for (int l = 0; l < n; ++l) {
      const DecodeStackLayer& L = a.layers[l0 + l];
      LayerParams& q = p.layer[l];
      if (encode_blocks(&q.w[kQkv], L.w_qkv, plan[kQkv]) || encode_blocks(&q.w[kO], L.w_o, plan[kO]) ||
          encode_blocks(&q.w[kGateUp], L.w_gate_up, plan[kGateUp]) || encode_blocks(&q.w[kDown], L.w_down, plan[kDown]))
        return cudaErrorInvalidValue;
      q.norm1 = static_cast<const __nv_bfloat16*>(L.norm1);
      q.norm2 = static_cast<const __nv_bfloat16*>(L.norm2);
      q.k_cache = static_cast<__nv_bfloat16*>(L.k_cache);
      q.v_cache = static_cast<__nv_bfloat16*>(L.v_cache);
    }
    decode_head_kernel<<<a.batch, 512, 0, stream>>>(p.x, p.layer[0].norm1, p.xn, a.hidden, a.eps,
                                                    reinterpret_cast<uint4*>(p.ss), (int)((lo.total - lo.ss) / 16));
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)a.num_sms);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemTotal;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kernel, p);
    if (e != cudaSuccess) return (int)e;
  }
  return cudaSuccess;
}

}  // namespace

int decode_stack_supported(int batch, int hidden, int ffn, int hq, int hkv, int head_dim, int s_max, int num_sms) {
  PhasePlan plan[4];
  Layout lo{};
  return make_plan(batch, hidden, ffn, hq, hkv, head_dim, s_max, num_sms, plan, lo) ? (int)cudaErrorInvalidValue : 0;
}

size_t decode_stack_scratch_bytes(int batch, int hidden, int ffn, int hq, int hkv, int head_dim, int s_max, int num_sms) {
  PhasePlan plan[4];
  Layout lo{};
  return make_plan(batch, hidden, ffn, hq, hkv, head_dim, s_max, num_sms, plan, lo) ? 0 : lo.total;
}

int launch_decode_stack(const DecodeStackArgs& a, cudaStream_t stream) {
  PhasePlan plan[4];
  Layout lo{};
  if (a.n_layers < 1 || make_plan(a.batch, a.hidden, a.ffn, a.hq, a.hkv, a.head_dim, a.s_max, a.num_sms, plan, lo))
    return cudaErrorInvalidValue;
  if (a.scratch_bytes < lo.total || ((uintptr_t)a.scratch | (uintptr_t)a.x | (uintptr_t)a.y) % 16 != 0 ||
      a.rope_theta <= 1.0f || (a.pos_dev == nullptr && (a.pos0 < 0 || a.pos0 >= a.s_max)))
    return cudaErrorInvalidValue;
  for (int l = 0; l < a.n_layers; ++l) {
    const DecodeStackLayer& L = a.layers[l];
    if (((uintptr_t)L.w_qkv | (uintptr_t)L.w_o | (uintptr_t)L.w_gate_up | (uintptr_t)L.w_down | (uintptr_t)L.norm1 |
         (uintptr_t)L.norm2 | (uintptr_t)L.k_cache | (uintptr_t)L.v_cache) % 16 != 0)
      return cudaErrorInvalidValue;
  }
  return a.head_dim == 128 ? launch_steps<128>(a, plan, lo, stream) : launch_steps<64>(a, plan, lo, stream);
}

}  // namespace smr
