// Rank-local GEMV on the tensor cores (tcgen05) for decode batches 1..16, with the element-wise work
// of a decode step folded into its two ends.  No upstream counterpart; the form with peers (sums
// exchanged inside the kernel) is gemv_allreduce_tc.cu.
//
//     out[b, n] = x[b, :] . W[n, :]          W stored [N, K] (K contiguous) or [K, N]
//
// What bounds it: the weights cross HBM once, and at decode batches nothing else is large.  A probe that
// only streams the weights by TMA (no math) reaches 7.1 TB/s and does not care how the rows are cut up as
// long as about a hundred CTAs pull on them; on top of that every launch pays about 3.7 us until its stream
// is up, as much as the whole 17-21 MB weight of a QKV or o-projection shard takes.  Hence:
//   * The product is computed transposed (128 weight rows = the MMA's M, the batch padded to 16 = its N), so
//     one elected thread feeds the tensor core and the SM's other warps only touch x and the result.
//   * Row tile and K split are chosen so that one wave of CTAs covers N as evenly as possible
//     (plan_gemv): the K splits of a tile are the CTAs of a cluster and meet in distributed shared memory.
//   * One 144 KB weight ring per CTA, filled before anything else happens.  Inside a decode step the kernel
//     is launched with programmatic stream serialization and `static_w`: the ring then fills while the
//     predecessor is still running, because the weights do not depend on it; x is only touched after
//     griddepcontrol.wait.  (Four chained GEMVs of a TP8 layer: 39.5 us without the overlap, 33.0 with.)
//   * x is written into shared memory by the four epilogue warps, which have nothing else to do until the
//     accumulator is complete.  On the way they can apply the RMSNorm that precedes a column-parallel
//     projection; on the way out they can apply SiLU(gate) * up or the residual add that follows, and
//     leave the sums of squares the next RMSNorm needs.  A decode layer is then five launches instead of
//     eight, none of which only moves activations.
//
// Arithmetic of the fused ends is that of the stand-alone kernels (layer_glue.cu): the norm rounds to bf16
// before and after the weight, the projection is rounded to bf16 before the residual add.  Sums of squares
// are added up in a fixed order (per CTA, then over the CTAs' slots), so results do not depend on timing.
// SiLU(gate) * up is taken on the fp32 accumulators.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "../device/mbarrier.cuh"
#include "../device/pdl.cuh"
#include "../device/tcgen05.cuh"
#include "../device/tcgen05_pair.cuh"
#include "../device/tma.cuh"
#include "../device/vec.cuh"
#include "../symm/driver_api.h"
#include "gemv_local.h"

namespace smr {

namespace {

constexpr int kMmaM = 128;        // weight rows per MMA; a tile may use fewer (the rest of D is ignored)
constexpr int kBatchN = 16;       // MMA N: the batch, rows beyond it are zero
constexpr int kBK = 64;           // k per block = one 128-byte swizzle row
constexpr int kUmmaK = 16;
constexpr int kThreads = 192;     // warp 0: weight stream, warp 1: MMA, warps 2..5: x in, result out
constexpr int kStageBlocks = 2;    // k blocks per ring stage
constexpr uint32_t kRingBytes = 9 * 16384;
constexpr int kMaxStages = 12;
constexpr int kGroupBlocks = 4;                                   // k blocks of x staged together
constexpr uint32_t kXBlockBytes = kBatchN * kBK * 2;              // 2 KB
constexpr uint32_t kXGroupBytes = kGroupBlocks * kXBlockBytes;    // 8 KB
constexpr int kXGroups = 4;
constexpr uint32_t kXOffset = kRingBytes;
constexpr uint32_t kNormOffset = kXOffset + kXGroups * kXGroupBytes;        // [kXGroups][4 warps][256] bf16
constexpr uint32_t kBarOffset = kNormOffset + kXGroups * 4 * 512;
constexpr uint32_t kNumBars = 2 * kMaxStages + 2 * kXGroups + 1;
constexpr uint32_t kSsOffset = kBarOffset + ((8 * kNumBars + 127) & ~127u);   // [8][16] fp32, then [16] scales
constexpr uint32_t kMiscOffset = kSsOffset + 9 * 16 * 4;
constexpr uint32_t kSmemTotal = kMiscOffset + 16 + 1024;
constexpr uint32_t kTmemCols = 32;
static_assert(kSmemTotal <= 232448, "shared memory limit exceeded");

// K blocks a CTA takes, in whole stages.
__host__ __device__ __forceinline__ int k_blocks_per_cta(int kb_total, int ksplit) {
  const int per = (kb_total + ksplit - 1) / ksplit;
  return (per + kStageBlocks - 1) / kStageBlocks * kStageBlocks;
}

struct GemvLocalParams {
  const __nv_bfloat16* x;          // [batch, K]
  __nv_bfloat16* out;              // [batch, N] ([batch, N / 2] with silu)
  int batch, K, N;
  int rows;                        // weight rows of a tile (multiple of 8, at most 128)
  int ksplit, stages;
  int deep_box;                    // one TMA load fills a stage (tensor map of encode_w_blocks)
  const __nv_bfloat16* norm_w;     // RMSNorm weight [K] applied to x, or nullptr
  const float* ss_in;              // [n_ss][16] partial sums of squares of x
  int n_ss;
  float eps;
  int silu;                        // rows of W: gate [0, N / 2), up [N / 2, N)
  const __nv_bfloat16* residual;   // [batch, N] added to the rounded product, or nullptr
  float* ss_out;                   // [gridDim.x][16] partial sums of squares of what is written, or nullptr
  int static_w;                    // the weights do not depend on earlier kernels of the stream
  uint64_t timeout_ns;
  Status* status;
};

// MN-major, 128-byte swizzle: 8-row k groups 1024 B apart (SBO), 64-element n groups 16 KB apart (LBO: a
// stage holds 128 k rows of columns 0..63 of the tile, then those of columns 64..127).
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((kStageBlocks * 8192u) >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)2u << 61;
  return d;
}

__device__ __forceinline__ void group_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_smem_addr, uint32_t cta) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(map_to_cta(local_smem_addr, cta)) : "memory");
  return v;
}

__device__ __forceinline__ float round_bf16(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

// Eight bf16 of x, normalised: bf16(bf16(x * scale) * w)
__device__ __forceinline__ Vec16 normed(const Vec16& x, const Vec16& w, float s) {
  auto two = [s](uint32_t a, uint32_t g) {
    return pack_bf16x2(round_bf16(bf16lo_to_f32(a) * s) * bf16lo_to_f32(g),
                       round_bf16(bf16hi_to_f32(a) * s) * bf16hi_to_f32(g));
  };
  return Vec16{two(x.x, w.x), two(x.y, w.y), two(x.z, w.z), two(x.w, w.w)};
}

template <bool kNK>
__global__ void __launch_bounds__(kThreads, 1)
gemv_local_kernel(const __grid_constant__ CUtensorMap tmap_w, const GemvLocalParams p) {
  extern __shared__ uint8_t smem_raw[];
  // the same offset in every CTA of the cluster: the dynamic window starts at the same shared address
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBarOffset);
  uint64_t* w_full = bars;
  uint64_t* w_empty = bars + kMaxStages;
  uint64_t* x_full = bars + 2 * kMaxStages;
  uint64_t* x_empty = bars + 2 * kMaxStages + kXGroups;
  uint64_t* tmem_full = bars + 2 * kMaxStages + 2 * kXGroups;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kMiscOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = (int)blockIdx.x / p.ksplit, kh = (int)blockIdx.x % p.ksplit;   // kh = rank in the cluster
  const int half = p.rows >> 1;                                    // silu: gate rows (= up rows) of the tile
  const int n0 = tile * (p.silu ? half : p.rows);                  // first output column of the tile
  const int n_out = p.silu ? p.N >> 1 : p.N;
  const uint32_t block_bytes = (uint32_t)p.rows * 128u;            // one k block
  const uint32_t stage_bytes = kStageBlocks * block_bytes;

  const int kb_total = (p.K + kBK - 1) / kBK;
  const int kb_per = k_blocks_per_cta(kb_total, p.ksplit);
  const int kb0 = kh * kb_per;
  const int n_kb = (kb0 + kb_per < kb_total ? kb0 + kb_per : kb_total) - kb0;     // may be <= 0
  const int n_groups = n_kb > 0 ? (n_kb + kGroupBlocks - 1) / kGroupBlocks : 0;

  const int n_steps = n_kb > 0 ? (n_kb + kStageBlocks - 1) / kStageBlocks : 0;    // ring stages to fill

  auto load_stage = [&](int i, int stage) {
    const int k = (kb0 + i * kStageBlocks) * kBK;
    uint8_t* sw = smem + (size_t)stage * stage_bytes;
    mbar_arrive_expect_tx(&w_full[stage], stage_bytes);
    if constexpr (kNK) {
      // A stage is [k block][row][64 k]; with silu the rows of a block are gate rows, then up rows.  What lies
      // beyond the tensor is zero or meets rows of D that nobody reads.
      if (p.deep_box) {
        tma_load_4d(sw, &tmap_w, &w_full[stage], 0, n0, 0, k / kBK);
      } else {
#pragma unroll
        for (int j = 0; j < kStageBlocks; ++j) {
          tma_load_2d(sw + j * block_bytes, &tmap_w, &w_full[stage], k + j * kBK, n0);
          if (p.silu) tma_load_2d(sw + j * block_bytes + (size_t)half * 128, &tmap_w, &w_full[stage], k + j * kBK, n_out + n0);
        }
      }
    } else {
      tma_load_2d(sw, &tmap_w, &w_full[stage], n0, k);             // 128 k x columns 0..63 of the tile
      tma_load_2d(sw + kStageBlocks * 8192, &tmap_w, &w_full[stage], n0 + 64, k);
    }
  };

  // Set-up: warp 0 initialises the barriers and goes straight on to the weight stream, warp 1 allocates tensor
  // memory, the others clear the rows of x beyond the batch, which stay zero for the whole kernel.
  const int etid = (int)threadIdx.x - 64;
  if (warp == 0) {
    for (int i = lane; i < (int)kNumBars; i += 32) mbar_init(&bars[i], &bars[i] >= x_full && &bars[i] < x_empty ? 128 : 1);
    mbar_fence_init();
    __syncwarp();
    asm volatile("bar.arrive 2, 192;" ::: "memory");
  } else {
    if (warp == 1) {
      tmem_alloc(tmem_slot, kTmemCols);
      tmem_relinquish_alloc_permit();
    } else {
      const int pad = (kBatchN - p.batch) * 8;                     // 16-byte chunks per block
      for (int i = etid; i < pad * kXGroups * kGroupBlocks; i += 128) {
        const int blk = i / pad, c = i - blk * pad;
        st_shared_16(smem_u32(smem + kXOffset) + (uint32_t)blk * kXBlockBytes + (uint32_t)p.batch * 128u + (uint32_t)c * 16u,
                     0u, 0u, 0u, 0u);
      }
    }
    tcgen05_fence_before_thread_sync();
    asm volatile("bar.sync 2, 192;" ::: "memory");
    tcgen05_fence_after_thread_sync();
  }
  bool failed = false;
  float* part = reinterpret_cast<float*>(smem);                    // [16][128] fp32 partial (ring idle by then)

  if (warp == 0) {
    if (elect_one()) {
      if (!p.static_w) pdl_wait();
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < n_steps; ++i) {
        if (i >= p.stages && !mbar_wait(&w_empty[stage], phase, p.timeout_ns)) {
          report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, stage, kWhereGemmEmpty);
          failed = true;
          break;
        }
        load_stage(i, stage);
        if (i == 0) pdl_launch_dependents();
        if (++stage == p.stages) { stage = 0; if (i >= p.stages) phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // kind::f16, bf16 x bf16 -> fp32, M = 128, N = 16; A MN-major (bit 15) when W is [K, N]
      constexpr uint32_t idesc = umma_idesc_bf16_f32(kMmaM, kBatchN) | (kNK ? 0u : (1u << 15));
      const uint32_t tmem_d = *tmem_slot;
      int stage = 0, xs = 0;
      uint32_t phase = 0, xphase = 0;
      for (int i = 0; i < n_steps; ++i) {
        const int in_group = i % (kGroupBlocks / kStageBlocks);
        if ((in_group == 0 && !mbar_wait(&x_full[xs], xphase, p.timeout_ns)) ||
            !mbar_wait(&w_full[stage], phase, p.timeout_ns)) {
          report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, stage, kWhereGemmFull);
          failed = true;
          break;
        }
        tcgen05_fence_after_thread_sync();
        const uint32_t sw = smem_u32(smem) + (uint32_t)stage * stage_bytes;
        const uint32_t sx = smem_u32(smem + kXOffset) + (uint32_t)xs * kXGroupBytes +
                            (uint32_t)in_group * kStageBlocks * kXBlockBytes;
#pragma unroll
        for (int j = 0; j < kStageBlocks; ++j) {
          // A, MN-major: +16 k rows = +2048 B; A, K-major and B: +16 k elements inside the 128-byte row = +32 B
          const uint64_t da = kNK ? umma_smem_desc_sw128(sw + (uint32_t)j * block_bytes) : desc_mn_sw128(sw + (uint32_t)j * 8192u);
          const uint64_t db = umma_smem_desc_sw128(sx + (uint32_t)j * kXBlockBytes);
          if (i * kStageBlocks + j < n_kb) {
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k)
              umma_bf16_ss(tmem_d, da + (kNK ? (uint64_t)(2 * k) : (uint64_t)(k * (2048 >> 4))), db + (uint64_t)(2 * k), idesc,
                           (i | j | k) != 0 ? 1u : 0u);
          }
        }
        umma_commit(&w_empty[stage]);
        if (in_group == kGroupBlocks / kStageBlocks - 1) {
          umma_commit(&x_empty[xs]);
          if (++xs == kXGroups) { xs = 0; xphase ^= 1; }
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (!failed) umma_commit(tmem_full);
    }
  } else {
    // ---------------- x into shared memory (normalised on the way when asked for) ----------------
    // Warp w takes rows w, w + 4, ... of the batch, a lane the same 16-byte chunk of each; cp.async puts a
    // chunk straight where the MMA reads it, and the thread that asked for it normalises it in place.
    // kXGroups groups are in flight: a group's latency (about 0.8 us from L2) is paid once, not per group.
    const int w4 = warp - 2;
    const uint32_t x_chunk = smem_u32(smem + kXOffset) + (uint32_t)(lane >> 3) * kXBlockBytes;
    const uint32_t g_chunk = smem_u32(smem + kNormOffset) + (uint32_t)w4 * 512u + (uint32_t)lane * 16u;
    auto chunk_at = [&](int slot, int b) {
      return x_chunk + (uint32_t)slot * kXGroupBytes + (uint32_t)b * 128u + (((uint32_t)(lane & 7) ^ (uint32_t)(b & 7)) << 4);
    };
    auto issue = [&](int grp) {
      const int slot = grp % kXGroups, k = (kb0 + grp * kGroupBlocks) * kBK + lane * 8;
      if (grp < n_groups) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int b = w4 + 4 * j;
          if (b < p.batch) {
            if (k < p.K) cp_async_16(chunk_at(slot, b), p.x + (size_t)b * p.K + k);
            else st_shared_16(chunk_at(slot, b), 0u, 0u, 0u, 0u);
          }
        }
        if (p.norm_w != nullptr && k < p.K && w4 < p.batch) cp_async_16(g_chunk + (uint32_t)slot * 2048u, p.norm_w + k);
      }
      cp_async_commit();                                           // an empty group keeps the count
    };
    pdl_wait();
    float scale[4] = {1.f, 1.f, 1.f, 1.f};
#pragma unroll
    for (int g = 0; g < kXGroups; ++g) issue(g);
    if (p.norm_w != nullptr) {
      float* red = reinterpret_cast<float*>(smem + kSsOffset);     // [8][16], then the 16 scales
      const int b = etid & 15, r = etid >> 4;
      float s = 0.f;
#pragma unroll 8
      for (int i = r; i < p.n_ss; i += 8) s += __ldcg(p.ss_in + i * 16 + b);
      red[r * 16 + b] = s;
      group_sync();
      if (etid < 16) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += red[i * 16 + etid];
        red[128 + etid] = rsqrtf(t / (float)p.K + p.eps);
      }
      group_sync();
#pragma unroll
      for (int j = 0; j < 4; ++j) scale[j] = red[128 + w4 + 4 * j];
    }
    uint32_t xphase = 0;
    for (int g = 0; g < n_groups; ++g) {
      const int slot = g % kXGroups;
      cp_async_wait<kXGroups - 2>();                               // group g is here (see the count of commits below)
      const bool in_k = (kb0 + g * kGroupBlocks) * kBK + lane * 8 < p.K;
      if (p.norm_w != nullptr && w4 < p.batch && in_k) {
        const Vec16 gw = ld_shared_16(g_chunk + (uint32_t)slot * 2048u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int b = w4 + 4 * j;
          if (b < p.batch) {
            const Vec16 v = normed(ld_shared_16(chunk_at(slot, b)), gw, scale[j]);
            st_shared_16(chunk_at(slot, b), v.x, v.y, v.z, v.w);
          }
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(&x_full[slot]);
      // Refill the slot of group g - 1, which the MMA thread has left or is about to leave: it can work on
      // group g meanwhile.  Commits so far at the top of iteration g: kXGroups + g - 1.
      if (g > 0) {
        const int back = (g - 1) % kXGroups;
        if (g - 1 + kXGroups < n_groups) {
          if (!mbar_wait(&x_empty[back], xphase, p.timeout_ns)) {
            if (lane == 0) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, back, kWhereGemmEmpty);
            failed = true;
            break;
          }
        }
        issue(g - 1 + kXGroups);
        if (back == kXGroups - 1) xphase ^= 1;
      }
    }
    cp_async_wait<0>();
    // ---------------- accumulator -> this CTA's shared memory ----------------
    const int quarter = warp & 3;
    const int col = quarter * 32 + lane;                           // tile row of W owned by this thread
    uint32_t acc[16];
#pragma unroll
    for (int b = 0; b < 16; ++b) acc[b] = 0u;
    if (n_kb > 0 && !failed) {
      if (!mbar_wait(tmem_full, 0, p.timeout_ns)) {
        if (lane == 0) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, 0, kWhereGemmTmemFull);
        failed = true;
      } else {
        tcgen05_fence_after_thread_sync();
        tmem_ld_32x32b_x16(*tmem_slot + ((uint32_t)(quarter * 32) << 16), acc);
        tmem_ld_wait();
      }
    }
#pragma unroll
    for (int b = 0; b < 16; ++b)
      if (b < p.batch) part[b * kMmaM + col] = __uint_as_float(acc[b]);
  }

  // ---- every partial of the tile is in its CTA's shared memory ----
  __syncwarp();
  cluster_sync_all();

  if (warp >= 2) {
    // ---------------- K reduction over the cluster, the fused end, the result ----------------
    // Warp w finishes batch rows w, w + 4, ...; a lane four consecutive columns of this CTA's share.
    const int quads = (p.silu ? half : p.rows) >> 2;
    const int q0 = kh * quads / p.ksplit, q1 = (kh + 1) * quads / p.ksplit;       // at most 32 of them
    const int c = (q0 + lane) * 4;
    const bool mine = q0 + lane < q1 && n0 + c < n_out;                           // n_out % 4 == 0
    const uint32_t part_addr = smem_u32(part);
    for (int b = warp - 2; b < p.batch; b += 4) {
      float ss = 0.f;
      if (mine) {
        const size_t at = (size_t)b * n_out + n0 + c;
        uint2 r2{0u, 0u};
        if (p.residual != nullptr) r2 = *reinterpret_cast<const uint2*>(p.residual + at);
        float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f), u4 = s4;
        for (int j = 0; j < p.ksplit; ++j) {                                      // split order: deterministic
          const float4 v = ld_cluster_f4(part_addr + (uint32_t)(b * kMmaM + c) * 4u, (uint32_t)j);
          s4.x += v.x; s4.y += v.y; s4.z += v.z; s4.w += v.w;
          if (p.silu) {
            const float4 u = ld_cluster_f4(part_addr + (uint32_t)(b * kMmaM + half + c) * 4u, (uint32_t)j);
            u4.x += u.x; u4.y += u.y; u4.z += u.z; u4.w += u.w;
          }
        }
        if (p.silu) {
          s4.x = s4.x / (1.0f + __expf(-s4.x)) * u4.x;
          s4.y = s4.y / (1.0f + __expf(-s4.y)) * u4.y;
          s4.z = s4.z / (1.0f + __expf(-s4.z)) * u4.z;
          s4.w = s4.w / (1.0f + __expf(-s4.w)) * u4.w;
        }
        if (p.residual != nullptr) {
          s4.x = round_bf16(s4.x) + bf16lo_to_f32(r2.x);
          s4.y = round_bf16(s4.y) + bf16hi_to_f32(r2.x);
          s4.z = round_bf16(s4.z) + bf16lo_to_f32(r2.y);
          s4.w = round_bf16(s4.w) + bf16hi_to_f32(r2.y);
        }
        uint2 o;
        o.x = pack_bf16x2(s4.x, s4.y);
        o.y = pack_bf16x2(s4.z, s4.w);
        if (!failed) *reinterpret_cast<uint2*>(p.out + at) = o;
        const float f0 = bf16lo_to_f32(o.x), f1 = bf16hi_to_f32(o.x), f2 = bf16lo_to_f32(o.y), f3 = bf16hi_to_f32(o.y);
        ss = f0 * f0 + f1 * f1 + f2 * f2 + f3 * f3;
      }
      if (p.ss_out != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) p.ss_out[(size_t)blockIdx.x * 16 + b] = ss;
      }
    }
  }

  if (__any_sync(0xffffffffu, failed)) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);               // let the loads in flight land
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  tcgen05_fence_after_thread_sync();
  if (warp == 1) tmem_dealloc(*tmem_slot, kTmemCols);
  // no CTA of the cluster leaves while another may still read its shared memory
  __syncwarp();
  cluster_sync_all();
}

int encode_w(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
             uint32_t box_outer) {
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {inner * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = DriverApi::get().cuTensorMapEncodeTiled(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1;
}

// W [N, K] seen as [K / 64][1 or 2 halves][rows of a half][64 k]: one box is kStageBlocks k blocks of a tile,
// each a complete K-major MMA operand (with two halves: gate rows, then the matching up rows).  K % 64 == 0.
int encode_w_blocks(CUtensorMap* map, const void* base, uint64_t K, uint64_t rows, uint64_t halves, uint32_t box_rows) {
  cuuint64_t dims[4] = {(cuuint64_t)kBK, rows, halves, K / kBK};
  cuuint64_t strides[3] = {K * 2, rows * K * 2, (cuuint64_t)kBK * 2};
  cuuint32_t box[4] = {(cuuint32_t)kBK, box_rows, (cuuint32_t)halves, (cuuint32_t)kStageBlocks};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = DriverApi::get().cuTensorMapEncodeTiled(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1;
}

// What the planner needs to know of a device, looked up once: how many clusters of 1, 2, 4 and 8 CTAs of
// this kernel are resident at once (GPCs do not all hold a multiple of the cluster size).
struct DeviceFit {
  int rc = -1;                // -1: not looked up yet, 0: fine, else a cudaError_t
  int clusters[4] = {0, 0, 0, 0};
};

template <bool kNK>
int device_fit(int dev, DeviceFit& fit) {
  auto kernel = gemv_local_kernel<kNK>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemTotal);
  int sms = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int i = 0; i < 4 && e == cudaSuccess; ++i) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(sms / (1 << i)) << i, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemTotal;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << i;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&fit.clusters[i], kernel, &cfg);
  }
  return (int)e;
}

const DeviceFit* fit_of_current_device(bool nk) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static DeviceFit fits[2][kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  DeviceFit& f = fits[nk ? 1 : 0][dev];
  std::lock_guard<std::mutex> lock(mu);
  if (f.rc < 0) f.rc = nk ? device_fit<true>(dev, f) : device_fit<false>(dev, f);
  return &f;
}

struct GemvPlan {
  int rows = kMmaM, ksplit = 1, tiles = 1;
};

// Row tile and K split: the pair whose busiest CTA has the least to do, counted as rows x k blocks x waves.
// Rows are cut to a multiple of 8 (the swizzle atom; 16 when gate and up share a tile) so that one wave covers
// N evenly: 8192 columns become 74 tiles of 112 rows x 2 K splits on 148 SMs.  A tcgen05.mma reads all 128
// rows of its A operand from shared memory however few belong to the tile (60 cycles for K = 16), so tiles
// below 96 rows cost as much as 96: K is split before N is cut finer.  A larger cluster has to win by 5 %
// to be worth its wider barrier.  W stored [K, N] comes in whole 128-column tiles.
GemvPlan plan_gemv(const DeviceFit& fit, int N, int K, bool nk, bool silu, int num_sms) {
  GemvPlan best;
  const int cols = silu ? N / 2 : N;
  const int kb_total = (K + kBK - 1) / kBK;
  double best_cost = 0;
  for (int i = 0; i < 4; ++i) {
    const int ks = 1 << i;
    if (ks > 1 && kb_total < kStageBlocks * ks) break;
    int clusters = fit.clusters[i] < num_sms / ks ? fit.clusters[i] : num_sms / ks;
    if (clusters < 1) break;
    const int most = silu ? kMmaM / 2 : kMmaM;
    int c = nk ? ((cols + clusters - 1) / clusters + 7) / 8 * 8 : most;
    if (c > most) c = most;
    const int tiles = (cols + c - 1) / c, waves = (tiles + clusters - 1) / clusters;
    const int rows = silu ? 2 * c : c;
    const double cost = (double)(rows < 96 ? 96 : rows) * k_blocks_per_cta(kb_total, ks) * waves;
    if (i == 0 || cost < 0.95 * best_cost) {
      best_cost = cost;
      best.rows = rows;
      best.ksplit = ks;
      best.tiles = tiles;
    }
  }
  return best;
}

}  // namespace

int gemv_local_ctas(int N, int K, bool weights_nk, bool silu, int num_sms) {
  const DeviceFit* fit = fit_of_current_device(weights_nk);
  if (fit == nullptr || fit->rc != 0) return -(int)(fit == nullptr ? cudaErrorInvalidDevice : (cudaError_t)fit->rc);
  const GemvPlan plan = plan_gemv(*fit, N, K, weights_nk, silu, num_sms);
  return plan.tiles * plan.ksplit;
}

int launch_gemv_local(const GemvLocalArgs& a, cudaStream_t stream) {
  if (a.batch < 1 || a.batch > kBatchN || a.N < 8 || a.K < 8 || a.N % 8 != 0 || a.K % 8 != 0 || a.num_sms < 1)
    return cudaErrorInvalidValue;
  const bool fused = a.norm_w != nullptr || a.silu || a.residual != nullptr || a.ss_out != nullptr;
  if (fused && !a.weights_nk) return cudaErrorInvalidValue;
  if (a.silu && (a.N % 16 != 0 || a.residual != nullptr)) return cudaErrorInvalidValue;
  if (a.norm_w != nullptr && (a.ss_in == nullptr || a.n_ss < 1)) return cudaErrorInvalidValue;
  if (((uintptr_t)a.x | (uintptr_t)a.w | (uintptr_t)a.norm_w) % 16 != 0 ||
      ((uintptr_t)a.out | (uintptr_t)a.residual) % 8 != 0)
    return cudaErrorInvalidValue;
  const DeviceFit* fit = fit_of_current_device(a.weights_nk);
  if (fit == nullptr) return cudaErrorInvalidDevice;
  if (fit->rc != 0) return fit->rc;
  const GemvPlan plan = plan_gemv(*fit, a.N, a.K, a.weights_nk, a.silu, a.num_sms);

  GemvLocalParams p{};
  p.x = static_cast<const __nv_bfloat16*>(a.x);
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.batch = a.batch; p.K = a.K; p.N = a.N;
  p.rows = plan.rows;
  p.ksplit = plan.ksplit;
  p.stages = (int)(kRingBytes / (kStageBlocks * (uint32_t)plan.rows * 128u));
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  p.norm_w = static_cast<const __nv_bfloat16*>(a.norm_w);
  p.ss_in = a.ss_in; p.n_ss = a.n_ss; p.eps = a.eps;
  p.silu = a.silu ? 1 : 0;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual);
  p.ss_out = a.ss_out;
  p.static_w = a.overlap && a.static_w ? 1 : 0;
  p.timeout_ns = a.timeout_ns;
  p.status = a.status;

  CUtensorMap tw;
  const uint32_t box_rows = (uint32_t)(a.silu ? plan.rows / 2 : plan.rows);
  p.deep_box = a.weights_nk && a.K % kBK == 0 ? 1 : 0;
  const int bad = p.deep_box     ? encode_w_blocks(&tw, a.w, (uint64_t)a.K, (uint64_t)(a.silu ? a.N / 2 : a.N), a.silu ? 2 : 1, box_rows)
                  : a.weights_nk ? encode_w(&tw, a.w, (uint64_t)a.K, (uint64_t)a.N, kBK, box_rows)
                                 : encode_w(&tw, a.w, (uint64_t)a.N, (uint64_t)a.K, 64, kStageBlocks * kBK);
  if (bad) return cudaErrorInvalidValue;

  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(plan.tiles * plan.ksplit), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)plan.ksplit;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.overlap ? 2 : 1;
  return (int)(a.weights_nk ? cudaLaunchKernelEx(&cfg, gemv_local_kernel<true>, tw, p)
                            : cudaLaunchKernelEx(&cfg, gemv_local_kernel<false>, tw, p));
}

}  // namespace smr
