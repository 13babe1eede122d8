// Rank-local GEMV and skinny GEMM on the tensor cores (tcgen05): 1 to 128 rows of x.  No upstream counterpart; the
// form with peers (sums exchanged inside the kernel) is gemv_allreduce_tc.cu.
//
//     out[b, n] = x[b, :] . W[n, :]          W stored [N, K] (K contiguous) or, up to 16 rows, [K, N]
//     optional ends: SiLU(gate) * up over two halves of W's rows, or a residual added to the rounded product
//
// What bounds it: the weights cross HBM once, and at these batches nothing else is large.  A probe that
// only streams the weights by TMA (no math) reaches 7.1 TB/s and does not care how the rows are cut up as
// long as about a hundred CTAs pull on them; on top of that every launch pays about 3.7 us until its stream
// is up, as much as the whole 17-21 MB weight of a QKV or o-projection shard takes.  Hence:
//   * The product is computed transposed (up to 128 weight rows = the MMA's M, the batch padded to 16, 32, 64 or 128 = its N), so
//     one elected thread feeds the tensor core, one fills the weight ring and one loads x.
//   * Row tile and K split are chosen so that one wave of CTAs covers N as evenly as possible
//     (plan_gemv): the K splits of a tile are the CTAs of a cluster and meet in distributed shared memory.
//   * One weight ring of 128 to 192 KB per CTA, filled before anything else happens.
//   * The issuing thread is the next limit: a k block of a 56-row tile arrives every 280 cycles.  MMAs of 64 rows where the
//     tile fits (23 cycles against 39 for 128), a fixed number of k blocks per stage, and the next stage's barrier
//     tested before this stage's MMAs go out: 155 cycles per block instead of 250.
//   * A tiled GEMM computes 256 rows however few there are, 0.28 us per K block and pair of SMs, which is half the speed
//     of HBM: 64 rows through 7168 x 8192 with SwiGLU took 36 us, here 25.  x is read by every CTA out of L2, so tiles
//     stay wide (128 weight rows and K splits) as the batch grows.
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

constexpr int kMaxRows = 128;     // weight rows of a tile (MMA M is 64 or 128; the rest of D is ignored)
constexpr int kBK = 64;           // k per block = one 128-byte swizzle row
constexpr int kUmmaK = 16;
constexpr int kThreads = 192;     // warp 0: weight stream, warp 1: MMA, warps 2..5: result (warp 2: x first)
constexpr int kStageBlocks = 2;    // k blocks per ring stage
constexpr int kMaxStages = 18;
constexpr uint32_t kOperandBytes = 14 * 16384;                    // the weight ring and, behind it, the ring of x
// BN: the batch, padded (the MMA's N); what lies in the rows beyond it only reaches columns of D that nobody reads.
template <int BN>
struct Cfg {
  static constexpr uint32_t kXBlockBytes = BN * kBK * 2;
  static constexpr int kGroupBlocks = BN <= 32 ? 4 : 2;           // k blocks of x under one barrier
  static constexpr int kXGroups = BN == 128 ? 3 : 4;
  static constexpr uint32_t kRingBytes = kOperandBytes - kXGroups * kGroupBlocks * kXBlockBytes;
  static constexpr uint32_t kTmemCols = BN < 32 ? 32 : BN;
};
constexpr int kMaxXGroups = 4;
constexpr uint32_t kBarOffset = kOperandBytes;
constexpr uint32_t kNumBars = 2 * kMaxStages + 2 * kMaxXGroups + 1;
constexpr uint32_t kMiscOffset = kBarOffset + ((8 * kNumBars + 15) & ~15u);
constexpr uint32_t kSmemTotal = kMiscOffset + 16 + 1024;
static_assert(kSmemTotal <= 232448, "shared memory limit exceeded");

// K blocks a CTA takes, in whole stages.
__host__ __device__ __forceinline__ int k_blocks_per_cta(int kb_total, int ksplit) {
  const int per = (kb_total + ksplit - 1) / ksplit;
  return (per + kStageBlocks - 1) / kStageBlocks * kStageBlocks;
}

struct GemvLocalParams {
  __nv_bfloat16* out;              // [batch, N]
  int batch, K, N;
  int rows;                        // weight rows of a tile (multiple of 8, at most 128)
  int ksplit, stages;
  int halves;                      // 2: a tile is rows / 2 gate rows and rows / 2 up rows, one output column each
  int interleaved;                 // with 2: 128 gate rows, then their 128 up rows, ...; else all gate, then all up
  const __nv_bfloat16* residual;   // [batch, N] or nullptr
  int deep_box;                    // one TMA load fills a stage (tensor map of encode_w_blocks)
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

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_smem_addr, uint32_t cta) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(map_to_cta(local_smem_addr, cta)) : "memory");
  return v;
}

template <int BN, bool kNK>
__global__ void __launch_bounds__(kThreads, 1)
gemv_local_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GemvLocalParams p) {
  using C = Cfg<BN>;
  constexpr int kGroupBlocks = C::kGroupBlocks, kXGroups = C::kXGroups;
  constexpr uint32_t kXOffset = C::kRingBytes, kXBlockBytes = C::kXBlockBytes;
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
  const int cols = p.rows / p.halves, n_out = p.N / p.halves;
  const int n0 = tile * cols;                                      // first output column of the tile
  const int row0 = p.interleaved ? (n0 >> 7) * 256 + (n0 & 127) : n0;   // its row of W
  const uint32_t block_bytes = (uint32_t)p.rows * 128u;            // one k block
  const uint32_t stage_bytes = kStageBlocks * block_bytes;

  const int kb_total = (p.K + kBK - 1) / kBK;
  const int kb_per = k_blocks_per_cta(kb_total, p.ksplit);
  const int kb0 = kh * kb_per;
  const int n_kb = (kb0 + kb_per < kb_total ? kb0 + kb_per : kb_total) - kb0;     // may be <= 0
  const int n_steps = n_kb > 0 ? (n_kb + kStageBlocks - 1) / kStageBlocks : 0;    // ring stages to fill

  auto load_stage = [&](int i, int stage) {
    const int k = (kb0 + i * kStageBlocks) * kBK;
    uint8_t* sw = smem + (size_t)stage * stage_bytes;
    mbar_arrive_expect_tx(&w_full[stage], stage_bytes);
    if constexpr (kNK) {
      // A stage is [k block][row][64 k].  What lies beyond the tensor is zero.
      if (p.deep_box) {
        tma_load_4d(sw, &tmap_w, &w_full[stage], 0, n0, k / kBK, 0);
      } else {
#pragma unroll
        for (int j = 0; j < kStageBlocks; ++j) {
          tma_load_2d(sw + j * block_bytes, &tmap_w, &w_full[stage], k + j * kBK, row0);
          if (p.halves == 2)
            tma_load_2d(sw + j * block_bytes + (size_t)cols * 128, &tmap_w, &w_full[stage], k + j * kBK,
                        row0 + (p.interleaved ? 128 : n_out));
        }
      }
    } else {
      tma_load_2d(sw, &tmap_w, &w_full[stage], n0, k);             // 128 k x columns 0..63 of the tile
      tma_load_2d(sw + kStageBlocks * 8192, &tmap_w, &w_full[stage], n0 + 64, k);
    }
  };

  // Set-up: warp 0 initialises the barriers and goes straight on to the weight stream, warp 1 allocates tensor memory.
  if (warp == 0) {
    for (int i = lane; i < (int)kNumBars; i += 32) mbar_init(&bars[i], 1);
    mbar_fence_init();
    __syncwarp();
    asm volatile("bar.arrive 2, 192;" ::: "memory");
  } else {
    if (warp == 1) {
      tmem_alloc(tmem_slot, C::kTmemCols);
      tmem_relinquish_alloc_permit();
    }
    tcgen05_fence_before_thread_sync();
    asm volatile("bar.sync 2, 192;" ::: "memory");
    tcgen05_fence_after_thread_sync();
  }
  bool failed = false;
  float* part = reinterpret_cast<float*>(smem);                    // [BN][128] fp32 partial (ring idle by then)

  if (warp == 0) {
    if (elect_one()) {
      pdl_wait();
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
      // kind::f16, bf16 x bf16 -> fp32, N = BN; A MN-major (bit 15) when W is [K, N].  A wait that runs out is remembered
      // and not acted upon, to keep the loop free of exits; k blocks beyond K are zero on both sides.
      const uint32_t idesc = umma_idesc_bf16_f32(p.rows <= 64 ? 64 : 128, BN) | (kNK ? 0u : (1u << 15));
      const uint32_t tmem_d = *tmem_slot;
      int stage = 0, xs = 0;
      uint32_t phase = 0, xphase = 0;
      bool w_ready = false, x_ready = false;
      for (int i = 0; i < n_steps; ++i) {
        const int in_group = i % (kGroupBlocks / kStageBlocks);
        if (in_group == 0 && !x_ready) failed |= !mbar_wait(&x_full[xs], xphase, failed ? 0 : p.timeout_ns);
        if (!w_ready) failed |= !mbar_wait(&w_full[stage], phase, failed ? 0 : p.timeout_ns);
        tcgen05_fence_after_thread_sync();
        const bool group_ends = in_group == kGroupBlocks / kStageBlocks - 1;
        const int stage1 = stage + 1 == p.stages ? 0 : stage + 1, xs1 = xs + 1 == kXGroups ? 0 : xs + 1;
        w_ready = i + 1 < n_steps && mbar_test(&w_full[stage1], phase ^ (stage1 == 0 ? 1u : 0u));
        x_ready = group_ends && i + 1 < n_steps && mbar_test(&x_full[xs1], xphase ^ (xs1 == 0 ? 1u : 0u));
        const uint32_t sw = smem_u32(smem) + (uint32_t)stage * stage_bytes;
        const uint32_t sx = smem_u32(smem + kXOffset) + (uint32_t)(xs * kGroupBlocks + in_group * kStageBlocks) * kXBlockBytes;
#pragma unroll
        for (int j = 0; j < kStageBlocks; ++j) {
          // A, MN-major: +16 k rows = +2048 B; A, K-major and B: +16 k elements inside the 128-byte row = +32 B
          const uint64_t da = kNK ? umma_smem_desc_sw128(sw + (uint32_t)j * block_bytes) : desc_mn_sw128(sw + (uint32_t)j * 8192u);
          const uint64_t db = umma_smem_desc_sw128(sx + (uint32_t)j * kXBlockBytes);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k)
            umma_bf16_ss(tmem_d, da + (kNK ? (uint64_t)(2 * k) : (uint64_t)(k * (2048 >> 4))), db + (uint64_t)(2 * k), idesc,
                         (i | j | k) != 0 ? 1u : 0u);
        }
        umma_commit(&w_empty[stage]);
        if (group_ends) {
          umma_commit(&x_empty[xs]);
          xs = xs1;
          if (xs1 == 0) xphase ^= 1;
        }
        stage = stage1;
        if (stage1 == 0) phase ^= 1;
      }
      if (failed) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, stage, kWhereGemmFull);
      umma_commit(tmem_full);
    }
  } else {
    pdl_wait();
    if (warp == 2) {
      // ---------------- x: k blocks of all batch rows, as many as the weight ring's stages hold ----------------
      if (elect_one()) {
        const int n = n_steps * kStageBlocks;
        for (int kb = 0, g = 0; kb < n; kb += kGroupBlocks, ++g) {
          const int slot = g % kXGroups, blocks = n - kb < kGroupBlocks ? n - kb : kGroupBlocks;
          if (g >= kXGroups && !mbar_wait(&x_empty[slot], (uint32_t)(g / kXGroups - 1) & 1u, p.timeout_ns)) {
            report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, slot, kWhereGemmEmpty);
            failed = true;
            break;
          }
          mbar_arrive_expect_tx(&x_full[slot], (uint32_t)(blocks * p.batch) * 128u);
          for (int j = 0; j < blocks; ++j)
            tma_load_2d(smem + kXOffset + (size_t)(slot * kGroupBlocks + j) * kXBlockBytes, &tmap_x, &x_full[slot],
                        (kb0 + kb + j) * kBK, 0);
        }
      }
      failed = __any_sync(0xffffffffu, failed);
    }
    if (p.residual != nullptr) {                                   // this tile of it into L2 while the weights stream in
      const int lines = (cols * 2 + 127) / 128 + 1;
      for (int i = (int)threadIdx.x - 64; i < lines * p.batch; i += 128) {
        const int b = i / lines, c = n0 + (i - b * lines) * 64;
        if (c < n_out) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.residual + (size_t)b * n_out + c));
      }
    }
    // ---------------- accumulator -> this CTA's shared memory ----------------
    const int quarter = warp & 3;
    // the tile row of W this thread owns: an MMA of 64 rows leaves sixteen of them in each quarter of the lanes
    const bool m64 = p.rows <= 64;
    const int col = m64 ? quarter * 16 + lane : quarter * 32 + lane;
    bool done = n_steps > 0 && !failed;                            // without k blocks the partial is zero
    if (done && !mbar_wait(tmem_full, 0, p.timeout_ns)) {
      if (lane == 0) report_status(p.status, kTimeoutMbarrier, 0, blockIdx.x, 0, kWhereGemmTmemFull);
      failed = true;
      done = false;
    }
    done = __all_sync(0xffffffffu, done);
    tcgen05_fence_after_thread_sync();
#pragma unroll
    for (int b0 = 0; b0 < BN; b0 += 16) {
      if (b0 >= p.batch) break;
      uint32_t acc[16];
#pragma unroll
      for (int b = 0; b < 16; ++b) acc[b] = 0u;
      if (done) {
        tmem_ld_32x32b_x16(*tmem_slot + ((uint32_t)(quarter * 32) << 16) + (uint32_t)b0, acc);
        tmem_ld_wait();
      }
      if (!m64 || lane < 16) {
#pragma unroll
        for (int b = 0; b < 16; ++b)
          if (b0 + b < p.batch) part[(b0 + b) * kMaxRows + col] = __uint_as_float(acc[b]);
      }
    }
  }

  // ---- every partial of the tile is in its CTA's shared memory ----
  __syncwarp();
  cluster_sync_all();

  if (warp >= 2) {
    // ---------------- K reduction over the cluster, the result ----------------
    // This CTA's share of the tile's columns in groups of four, a thread each; as many rows at once as the 128 threads
    // cover (with a row per warp 28 of 32 lanes were idle at eight K splits: 512 x 512 with 128 rows took 13.6 us, now
    // 6.2).  The parts of an item are all in flight at once.
    const int quads = cols >> 2;
    const int q0 = kh * quads / p.ksplit, nq = (kh + 1) * quads / p.ksplit - q0;  // may be 0
    const uint32_t part_addr = smem_u32(part);
    auto total = [&](int b, int row) {
      const uint32_t at = part_addr + (uint32_t)(b * kMaxRows + row) * 4u;
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < p.ksplit) v[j] = ld_cluster_f4(at, (uint32_t)j);
      float4 s4 = v[0];
#pragma unroll
      for (int j = 1; j < 8; ++j)                                                 // split order: deterministic
        if (j < p.ksplit) { s4.x += v[j].x; s4.y += v[j].y; s4.z += v[j].z; s4.w += v[j].w; }
      return s4;
    };
    auto silu = [](float g) { return g / (1.0f + __expf(-g)); };
    int width_log = 0;                                                            // of a row, in threads
    while ((1 << width_log) < nq) ++width_log;
    const int etid = (int)threadIdx.x - 64, q = etid & ((1 << width_log) - 1), c = (q0 + q) * 4;
    const bool mine = q < nq && n0 + c < n_out && !failed;                        // n_out % 4 == 0
#pragma unroll 2
    for (int b = etid >> width_log; mine && b < p.batch; b += 128 >> width_log) {
      const size_t at = (size_t)b * n_out + n0 + c;
      uint2 r{0u, 0u};
      if (p.residual != nullptr) r = *reinterpret_cast<const uint2*>(p.residual + at);
      float4 s4 = total(b, c);
      if (p.halves == 2) {
        const float4 u4 = total(b, cols + c);
        s4 = make_float4(silu(s4.x) * u4.x, silu(s4.y) * u4.y, silu(s4.z) * u4.z, silu(s4.w) * u4.w);
      }
      uint2 o = make_uint2(pack_bf16x2(s4.x, s4.y), pack_bf16x2(s4.z, s4.w));
      if (p.residual != nullptr)
        o = make_uint2(pack_bf16x2(bf16lo_to_f32(o.x) + bf16lo_to_f32(r.x), bf16hi_to_f32(o.x) + bf16hi_to_f32(r.x)),
                       pack_bf16x2(bf16lo_to_f32(o.y) + bf16lo_to_f32(r.y), bf16hi_to_f32(o.y) + bf16hi_to_f32(r.y)));
      *reinterpret_cast<uint2*>(p.out + at) = o;
    }
  }

  if (__any_sync(0xffffffffu, failed)) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);               // let the loads in flight land
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  tcgen05_fence_after_thread_sync();
  if (warp == 1) tmem_dealloc(*tmem_slot, C::kTmemCols);
  // no CTA of the cluster leaves while another may still read its shared memory
  __syncwarp();
  cluster_sync_all();
}

int encode_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
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

// W [N, K] seen as [K / 64][N][64 k]: one box is kStageBlocks k blocks of a tile, each a complete K-major MMA
// operand.  K % 64 == 0.
int encode_w_blocks(CUtensorMap* map, const void* base, uint64_t K, uint64_t rows, uint32_t box_rows) {
  cuuint64_t dims[4] = {(cuuint64_t)kBK, rows, K / kBK, 1};
  cuuint64_t strides[3] = {K * 2, (cuuint64_t)kBK * 2, rows * K * 2};
  cuuint32_t box[4] = {(cuuint32_t)kBK, box_rows, (cuuint32_t)kStageBlocks, 1};
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

int device_fit(const void* kernel, int dev, DeviceFit& fit) {
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

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const GemvLocalParams);
constexpr Kernel kKernels[] = {gemv_local_kernel<16, false>, gemv_local_kernel<16, true>, gemv_local_kernel<32, true>,
                               gemv_local_kernel<64, true>, gemv_local_kernel<128, true>};
constexpr int kNumKernels = 5;
constexpr int kPadded[kNumKernels] = {16, 16, 32, 64, 128};
constexpr uint32_t kRings[kNumKernels] = {Cfg<16>::kRingBytes, Cfg<16>::kRingBytes, Cfg<32>::kRingBytes,
                                          Cfg<64>::kRingBytes, Cfg<128>::kRingBytes};
int kernel_for(int batch, bool nk) { return !nk ? 0 : (batch <= 16 ? 1 : batch <= 32 ? 2 : batch <= 64 ? 3 : 4); }

const DeviceFit* fit_of_current_device(int which) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static DeviceFit fits[kNumKernels][kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  DeviceFit& f = fits[which][dev];
  std::lock_guard<std::mutex> lock(mu);
  if (f.rc < 0) f.rc = device_fit(reinterpret_cast<const void*>(kKernels[which]), dev, f);
  return &f;
}

struct GemvPlan {
  int rows = kMaxRows, ksplit = 1, tiles = 1;
};

// Row tile and K split: the pair whose busiest CTA has the least to do, counted as cycles per k block x k blocks plus
// 5000 (set-up, the first loads' latency, the reduction) for each wave: without these 5176 columns stored [1584, N]
// went in three waves of eight K splits, 14.7 us, now 6.4 in one of two.
// A k block costs the SM's share of HBM for its weight rows (25 bytes a cycle), its share of L2 for the weight rows and x
// (45), and the issuing thread 155 cycles or, at 64 rows of x and more, two for each of them.  Rows of W that do not
// start on 128-byte lines come in box by box, and tiles below 96 rows then cost as much as 96 where K is long: 6912 x
// 7048 24.4 -> 20.4 us, 3000 x 5000 11.3 -> 9.6 (below the line 960 x 1248 would lose, 4.3 -> 4.7).
// Rows are cut to a multiple of 8 (the swizzle atom) so that one wave covers N evenly: at batch 16, 8192 columns become
// 147 tiles of 56 rows on 148 SMs.  With gate and up a tile has half the columns, and where they alternate in groups
// of 128 it must not straddle one.  A larger cluster has to win by 5 % to be worth its wider barrier.  W stored [K, N]
// comes in whole 128-column tiles.
GemvPlan plan_gemv(const DeviceFit& fit, int batch, int padded, int N, int K, bool nk, int halves, bool interleaved, int num_sms) {
  GemvPlan best;
  const int kb_total = (K + kBK - 1) / kBK, n_out = N / halves;
  const bool narrow_costs = nk && K % kBK != 0 && K >= 1536;
  double best_cost = 0, best_work = 0;
  for (int i = 0; i < 4; ++i) {
    const int ks = 1 << i;
    if (ks > 1 && kb_total < kStageBlocks * ks) break;
    int clusters = fit.clusters[i] < num_sms / ks ? fit.clusters[i] : num_sms / ks;
    if (clusters < 1) break;
    int cols = nk ? ((n_out + clusters - 1) / clusters + 7) / 8 * 8 : kMaxRows;
    if (cols > kMaxRows / halves) cols = kMaxRows / halves;
    if (interleaved) cols = cols <= 16 ? 16 : (cols <= 32 ? 32 : 64);
    const int rows = cols * halves, tiles = (n_out + cols - 1) / cols, waves = (tiles + clusters - 1) / clusters;
    double per = (narrow_costs && rows < 96 ? 96 : rows) * 128 / 25.0;
    const double l2 = (rows + batch) * 128 / 45.0, issue = padded < 64 ? 155.0 : 30.0 + 2.0 * padded;
    if (l2 > per) per = l2;
    if (issue > per) per = issue;
    const double work = per * k_blocks_per_cta(kb_total, ks) * waves, cost = work + 5000.0 * waves;
    if (i == 0 || cost < best_cost - 0.05 * best_work) {
      best_cost = cost;
      best_work = work;
      best.rows = rows;
      best.ksplit = ks;
      best.tiles = tiles;
    }
  }
  return best;
}

}  // namespace

int launch_gemv_local(const GemvLocalArgs& a, cudaStream_t stream) {
  if (a.batch < 1 || a.batch > (a.weights_nk ? 128 : 16) || a.N < 8 || a.K < 8 || a.N % 8 != 0 || a.K % 8 != 0 || a.num_sms < 1)
    return cudaErrorInvalidValue;
  if (((uintptr_t)a.x | (uintptr_t)a.w) % 16 != 0 || (uintptr_t)a.out % 8 != 0) return cudaErrorInvalidValue;
  const int halves = a.epilogue != 0 ? 2 : 1;
  if (a.epilogue < 0 || a.epilogue > 2 || (a.epilogue != 0 && (!a.weights_nk || a.residual != nullptr)) ||
      a.N % (a.epilogue == 1 ? 256 : 8 * halves) != 0 || (uintptr_t)a.residual % 8 != 0)
    return cudaErrorInvalidValue;
  const int which = kernel_for(a.batch, a.weights_nk);
  const DeviceFit* fit = fit_of_current_device(which);
  if (fit == nullptr) return cudaErrorInvalidDevice;
  if (fit->rc != 0) return fit->rc;
  const GemvPlan plan = plan_gemv(*fit, a.batch, kPadded[which], a.N, a.K, a.weights_nk, halves, a.epilogue == 1, a.num_sms);

  GemvLocalParams p{};
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.batch = a.batch; p.K = a.K; p.N = a.N;
  p.rows = plan.rows;
  p.ksplit = plan.ksplit;
  p.stages = (int)(kRings[which] / (kStageBlocks * (uint32_t)plan.rows * 128u));
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  p.halves = halves;
  p.interleaved = a.epilogue == 1 ? 1 : 0;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual);
  p.timeout_ns = a.timeout_ns;
  p.status = a.status;

  CUtensorMap tw, tx;
  p.deep_box = a.weights_nk && halves == 1 && a.K % kBK == 0 ? 1 : 0;
  const int bad = p.deep_box     ? encode_w_blocks(&tw, a.w, (uint64_t)a.K, (uint64_t)a.N, (uint32_t)plan.rows)
                  : a.weights_nk ? encode_2d(&tw, a.w, (uint64_t)a.K, (uint64_t)a.N, kBK, (uint32_t)(plan.rows / halves))
                                 : encode_2d(&tw, a.w, (uint64_t)a.N, (uint64_t)a.K, 64, kStageBlocks * kBK);
  if (bad || encode_2d(&tx, a.x, (uint64_t)a.K, (uint64_t)a.batch, kBK, (uint32_t)a.batch)) return cudaErrorInvalidValue;

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
  return (int)cudaLaunchKernelEx(&cfg, kKernels[which], tw, tx, p);
}

}  // namespace smr
