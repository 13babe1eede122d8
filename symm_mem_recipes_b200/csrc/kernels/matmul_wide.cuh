// The GEMM of ag_matmul_2cta_sm100.cu without a gather for problems of at least one full wave: a CTA pair multiplies two
// neighbouring 256 x 256 tiles of a row at once, so that both share their rows of A.
//
// What bounds it: power.  In a loop of calls the 1000 W limit sets the clock (1050 to 1250 MHz of 1965 with one tile at
// a time), so what counts is the energy of a flop and not the cycles.  Two tiles at once load 96 KB per 2 x 256 x 256 x 64
// products instead of 128 (A once), and the tensor core takes A from its operand buffer for the second MMA
// (`.collector::a`, 0.5 %).  Energy per flop at 16384 x 3584 x 8192, one tile of 128 columns at a time: 0.86 pJ, 192
// columns 0.81, 256 columns 0.76, here 0.72.  At the full clock (operands of zeros) it takes 462 us against 458; a single
// call after a pause is no slower than one tile at a time (see plan_wide_units).
//
// Both accumulators (2 x 256 columns) fill TMEM, so there is no spare one to write while a tile is read.  Instead the two
// are skewed against one another (kSkew): at either end of the K loop the first gets a few K blocks alone and the
// second the same blocks after it.  Beside the MMAs an accumulator takes 2000 to 3000 cycles to read and as many to
// pass through shared memory, and a unit's end costs about 4000 cycles; both accumulators taken into registers before
// anything is stored, stores by the lanes instead of by TMA, stores spread over the next K loop, and 2 or 4 blocks
// of skew measured the same or worse.
//
// The shared-memory ring is dealt out in chunks of 16 KB (128 rows of 128 bytes): a K block of a wide unit takes
// three (A, B, B of the second tile), one of a single tile two, so that the tiles that fill no whole wave of wide
// units (and the K parts of the last ones) have the six stages in flight they need.  Chunks are given back in the
// order of the K blocks, so a barrier per K block in flight and a count of free chunks are enough.
#pragma once
#include <type_traits>

#include "../device/pdl.cuh"
#include "../device/tcgen05_pair.cuh"
#include "ag_matmul_common.cuh"

namespace smr {
namespace wide {

using namespace agmm;

constexpr int kBN = 256;                                         // columns of a tile
constexpr int kChunks = 12;                                      // of the ring
constexpr uint32_t kChunkBytes = kBM * kBK * 2;
constexpr int kInFlight = 8;                                     // K blocks in flight at most (kChunks / 2), a power of two
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kBoxBytes = 32 * 128;                         // of an epilogue warp: 32 rows x 128 bytes
constexpr uint32_t kBoxOffset = kChunks * kChunkBytes;
constexpr uint32_t kBarOffset = kBoxOffset + kEpiWarps * kBoxBytes;
constexpr uint32_t kNumBars = 2 * kInFlight + 4 + kEpiWarps;
constexpr uint32_t kSmemBytes = kBarOffset + 8 * kNumBars + 16 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory limit exceeded");
static_assert(kInFlight >= kChunks / 2, "a barrier per K block in flight");

// Place of a K block in the ring: its first chunk, and its barriers.
struct Cursor {
  uint32_t chunk = 0, bar = 0, phase = 0;
  __device__ __forceinline__ void next(int chunks) {
    chunk += (uint32_t)chunks;
    if (chunk >= (uint32_t)kChunks) chunk -= kChunks;
    if (++bar == kInFlight) { bar = 0; phase ^= 1; }
  }
};
__device__ __forceinline__ uint32_t chunk_at(uint32_t first, int i) {
  const uint32_t c = first + (uint32_t)i;
  return c >= (uint32_t)kChunks ? c - kChunks : c;
}

// kSwiGlu, kResidual: as in ag_matmul_2cta_kernel.  kTraced: an instantiation of its own fills p.trace (ag_trace::), so that
// the waits of the others are not timed.
template <bool kSwiGlu, bool kResidual, bool kTraced>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
matmul_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                   const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_residual, const AgMatmulParams p) {
  static_assert(!kResidual || !kSwiGlu, "the residual belongs to the plain epilogue");
  extern __shared__ uint8_t smem_raw[];
  // same offset in both CTAs: the dynamic window starts at the same shared address
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kBarOffset);   // leader: the bytes of both CTAs
  uint64_t* empty_bar = full_bar + kInFlight;
  uint64_t* tmem_full = empty_bar + kInFlight;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* residual_full = tmem_empty + 2;                      // of each epilogue warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(residual_full + kEpiWarps);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kInFlight; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2 * kEpiWarps);                  // used in the leader
    }
    for (int w = 0; w < kEpiWarps; ++w) mbar_init(&residual_full[w], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  cluster_sync_all();                 // barriers of both CTAs initialised, TMEM allocated
  tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();

  const int pair = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;
  const int n_pair_rows = (p.n_blocks_m + 1) >> 1, total_tiles = n_pair_rows * p.n_tiles_n;
  const int k_blocks = (p.K + kBK - 1) / kBK;
  bool failed = false;
  [[maybe_unused]] uint64_t* trc = kTraced ? p.trace + (size_t)blockIdx.x * ag_trace::kTraceSlots : nullptr;
  if (kTraced && threadIdx.x == 0) trc[ag_trace::kStart] = globaltimer_ns();
  // a wait on a barrier, with its time added to `total`
  auto timed_wait = [&p](uint64_t* bar, uint32_t parity, [[maybe_unused]] uint64_t& total) {
    if constexpr (kTraced) {
      const uint64_t t0 = globaltimer_ns();
      const bool ok = mbar_wait(bar, parity, p.timeout_ns);
      total += globaltimer_ns() - t0;
      return ok;
    } else {
      return mbar_wait(bar, parity, p.timeout_ns);
    }
  };

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      Cursor at, oldest;                                         // oldest: the next K block to come back
      int free = kChunks, wide_left = p.wide_units / n_pairs * k_blocks;   // K blocks of three chunks not yet back
      WideWork w;
      uint64_t t_stage = 0;
      pdl_wait();
      for (int wi = 0; !failed && wide_work(p, pair, n_pairs, total_tiles, k_blocks, wi, w); ++wi) {
        int prow, ni;
        work_coords(p, n_pair_rows, w.tile, w.halves, prow, ni);
        const int row0 = (prow * 2 + (int)cta_rank) * kBM;       // rows past M (an odd tail) read as zero
        const int b0 = ni * p.b_step + (int)cta_rank * p.b_pair, need = w.halves + 1;
#pragma unroll 1
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          while (free < need) {
            if (!timed_wait(&empty_bar[oldest.bar], oldest.phase, t_stage)) {
              report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, oldest.bar, kWhereGemmEmpty);
              failed = true;
              break;
            }
            const int back = wide_left > 0 ? 3 : 2;
            --wide_left;
            free += back;
            oldest.next(back);
          }
          if (failed) break;
          free -= need;
          if (leader) mbar_arrive_expect_tx(&full_bar[at.bar], 2u * (uint32_t)need * kChunkBytes);
          const uint32_t full_leader = map_to_cta(smem_u32(&full_bar[at.bar]), 0);
          auto chunk = [&](int i) { return smem + (size_t)chunk_at(at.chunk, i) * kChunkBytes; };
          tma_load_2d_pair(chunk(0), &tmap_a, full_leader, kb * kBK, row0);
          tma_load_2d_pair(chunk(1), &tmap_b, full_leader, kb * kBK, b0);
          if (w.halves == 2) tma_load_2d_pair(chunk(2), &tmap_b, full_leader, kb * kBK, b0 + p.b_step);
          at.next(need);
        }
      }
      if constexpr (kTraced) trc[ag_trace::kStageWait] = t_stage;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (leader && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16_f32(2 * kBM, kBN);
      constexpr int kSkew = 3;                                   // of the ring's four wide K blocks
      Cursor at;
      uint32_t acc = 0, acc_phase = 0;
      WideWork w;
      uint64_t t_operand = 0, t_tmem = 0;
      auto wait_operands = [&](const Cursor& c) {
        if (!timed_wait(&full_bar[c.bar], c.phase, t_operand)) {
          report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, c.bar, kWhereGemmFull);
          failed = true;
          return false;
        }
        tcgen05_fence_after_thread_sync();
        return true;
      };
      auto wait_accumulator = [&](uint32_t which, uint32_t parity) {
        if (!timed_wait(&tmem_empty[which], parity, t_tmem)) {
          report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, which, kWhereGemmTmemEmpty);
          failed = true;
          return false;
        }
        tcgen05_fence_after_thread_sync();
        return true;
      };
      auto operand = [&](const Cursor& c, int i) {
        return umma_smem_desc_sw128(smem_u32(smem) + chunk_at(c.chunk, i) * kChunkBytes);
      };
      // A K block into one accumulator (`b`: the chunk of B).
      auto multiply = [&](const Cursor& c, int b, uint32_t d, bool first) {
        const uint64_t da = operand(c, 0), db = operand(c, b);
#pragma unroll
        for (int k = 0; k < kBK / kUmmaK; ++k)
          umma_ss_pair<false>(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (!first || k != 0) ? 1u : 0u);
      };
      for (int wi = 0; !failed && wide_work(p, pair, n_pairs, total_tiles, k_blocks, wi, w); ++wi) {
        if (!wait_accumulator(acc, acc_phase ^ 1)) break;
        const uint32_t d0 = tmem_base + acc * 256u, d1 = tmem_base + (acc ^ 1) * 256u;
        if (w.halves == 1) {
#pragma unroll 1
          for (int kb = w.kb0; kb < w.kb1 && wait_operands(at); ++kb) {
            multiply(at, 1, d0, kb == w.kb0);
            umma_commit_pair(&empty_bar[at.bar]);
            at.next(2);
          }
          if (failed) break;
          umma_commit_pair(&tmem_full[acc]);
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1;
          continue;
        }
        const int head = k_blocks < kSkew ? k_blocks : kSkew, mid = k_blocks - kSkew > head ? k_blocks - kSkew : head;
        // K blocks [kb0, kb1) into the first accumulator, then into the second.
        auto apart = [&](int kb0, int kb1) {
          Cursor c = at;
#pragma unroll 1
          for (int kb = kb0; kb < kb1; ++kb, c.next(3)) {
            if (!wait_operands(c)) return;
            multiply(c, 1, d0, kb == 0);
          }
          if (kb1 == k_blocks) umma_commit_pair(&tmem_full[acc]);
          if (kb0 == 0 && !wait_accumulator(acc ^ 1, acc == 0 ? acc_phase ^ 1 : acc_phase)) return;
#pragma unroll 1
          for (int kb = kb0; kb < kb1; ++kb, at.next(3)) {
            multiply(at, 2, d1, kb == 0);
            umma_commit_pair(&empty_bar[at.bar]);
          }
        };
        apart(0, head);
#pragma unroll 1
        for (int kb = head; !failed && kb < mid && wait_operands(at); ++kb, at.next(3)) {
          const uint64_t da = operand(at, 0), db0 = operand(at, 1), db1 = operand(at, 2);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            umma_ss_pair<false, CollectA::kFill>(d0, da + (uint64_t)(2 * k), db0 + (uint64_t)(2 * k), idesc, 1u);
            umma_ss_pair<false, CollectA::kLastUse>(d1, da + (uint64_t)(2 * k), db1 + (uint64_t)(2 * k), idesc, 1u);
          }
          umma_commit_pair(&empty_bar[at.bar]);
        }
        if (!failed && mid < k_blocks) apart(mid, k_blocks);
        if (failed) break;
        umma_commit_pair(&tmem_full[acc ^ 1]);
        acc_phase ^= 1;
      }
      if constexpr (kTraced) {
        trc[ag_trace::kTmemWait] = t_tmem;
        trc[ag_trace::kOperandWait] = t_operand;
      }
    }
  } else {
    // ---------------- epilogue (eight warps of both CTAs) ----------------
    // A warp has 32 rows and one half of the columns of every tile.  It takes them into registers with all loads in flight
    // (one that waits by itself takes 700 cycles beside the MMAs), returns the accumulator, and sends them through
    // its box of shared memory (128-byte swizzle, see ag_matmul_2cta_kernel) by TMA.
    const int quarter = warp & 3, side = (warp - 2) >> 2;
    constexpr int kBoxes = kSwiGlu ? 1 : 2;                      // of a warp and tile
    constexpr int kOutCols = kSwiGlu ? kBN / 2 : kBN, kBoxCols = kOutCols / 2 / kBoxes;
    const int n_out = kSwiGlu ? p.N >> 1 : p.N;
    uint8_t* box = smem + kBoxOffset + (size_t)(side * 4 + quarter) * kBoxBytes;
    const uint32_t rowaddr = smem_u32(box) + (uint32_t)lane * 128u, sw = (uint32_t)(lane & 7);
    uint32_t acc = 0, acc_phase = 0;
    [[maybe_unused]] uint32_t residual_phase = 0;
    pdl_wait();
    const bool records = kTraced && warp == 2 && lane == 0;
    uint64_t t_acc = 0;
    [[maybe_unused]] uint64_t n_tiles = 0;
    if (records) trc[ag_trace::kEntered] = globaltimer_ns();
    WideWork w;
    w.halves = 1;
    for (int wi = 0, half = 1;; ++half) {
      if (half >= w.halves) {
        if (!wide_work(p, pair, n_pairs, total_tiles, k_blocks, wi++, w)) break;
        half = 0;
      }
      int prow, ni;
      work_coords(p, n_pair_rows, w.tile, w.halves, prow, ni);
      const int row0 = (prow * 2 + (int)cta_rank) * kBM + quarter * 32, col0 = (ni + half) * kOutCols + side * (kOutCols / 2);
      const bool stores = w.part < 0 && row0 < p.M;
      [[maybe_unused]] auto load_residual = [&](int b) {         // one lane
        bulk_wait_group_read<0>();                               // the store before has read the box
        mbar_arrive_expect_tx(&residual_full[warp - 2], kBoxBytes);
        tma_load_2d(box, &tmap_residual, &residual_full[warp - 2], col0 + b * kBoxCols, row0);
      };
      if constexpr (kResidual) {
        if (stores && lane == 0 && col0 < n_out) {
          load_residual(0);
          if (half == 0)
            for (int c = 1; c < 2 * w.halves; ++c) {
              const int col = col0 + (c >> 1) * kOutCols + (c & 1) * kBoxCols;
              if (col < n_out) tma_prefetch_2d(&tmap_residual, col, row0);
            }
        }
      }
      if (!timed_wait(&tmem_full[acc], acc_phase, t_acc)) {
        if (lane == 0) report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, acc, kWhereGemmTmemFull);
        failed = true;
        break;
      }
      if constexpr (kTraced) ++n_tiles;
      tcgen05_fence_after_thread_sync();
      const uint32_t taddr = tmem_base + acc * 256u + ((uint32_t)(quarter * 32) << 16);
      auto release_accumulator = [&] {
        tcgen05_fence_before_thread_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));
      };
      uint32_t word[kBoxes * 32];
      if (w.part >= 0) {
        // ---- split-K tail: park the fp32 partial for merge_tail_kernel ----
        float* mine = p.tail_scratch + (((size_t)w.tail_idx * p.tail_splits + w.part) * 2 + cta_rank) * ((size_t)kBM * kBN) +
                      (quarter * 32 + lane) * 4;
#pragma unroll 1
        for (int c = side * (kBN / 64); c < (side + 1) * (kBN / 64); ++c) {
          uint32_t v[32];
          if (w.kb1 > w.kb0) {
            tmem_ld_32x32b_x32(taddr + (uint32_t)(c * 32), v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = 0u;
          }
#pragma unroll
          for (int q = 0; q < 8; ++q)
            st_16(mine + (size_t)(c * 8 + q) * (kBM * 4), Vec16{v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]});
        }
        release_accumulator();
      } else {
        uint32_t v[4][32];                                       // pieces of 32 columns; SwiGLU: gate, gate, up, up
#pragma unroll
        for (int c = 0; c < 4; ++c)
          tmem_ld_32x32b_x32(taddr + (uint32_t)(kSwiGlu ? (c >> 1) * (kBN / 2) + side * 64 + (c & 1) * 32 : side * 128 + c * 32), v[c]);
        tmem_ld_wait();
        release_accumulator();
#pragma unroll
        for (int c = 0; c < 2 * kBoxes; ++c) {
          auto f = [&](int i) {
            float x = __uint_as_float(v[c][i]);
            if constexpr (kSwiGlu) x = x / (1.0f + __expf(-x)) * __uint_as_float(v[c + 2][i]);
            return x;
          };
#pragma unroll
          for (int i = 0; i < 16; ++i) word[c * 16 + i] = pack_bf16x2(f(2 * i), f(2 * i + 1));
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
      if (!stores) continue;
#pragma unroll
      for (int b = 0; b < kBoxes; ++b) {
        const int col = col0 + b * kBoxCols;
        if (col < n_out) {
          if constexpr (kResidual) {
            if (b > 0 && lane == 0) load_residual(b);
            if (!mbar_wait(&residual_full[warp - 2], residual_phase, p.timeout_ns)) {
              if (lane == 0) report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, b, kWhereGemmFull);
              failed = true;
            }
            residual_phase ^= 1u;
          } else {
            if (lane == 0) bulk_wait_group_read<0>();            // the store before has read the box
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* q = word + b * 32 + j * 4;
            Vec16 o{q[0], q[1], q[2], q[3]};
            const uint32_t chunk = rowaddr + (((uint32_t)j ^ sw) << 4);
            if constexpr (kResidual) o = add_bf16x8(o, ld_shared_16(chunk));
            st_shared_16(chunk, o.x, o.y, o.z, o.w);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmap_c, box, col, row0);
            bulk_commit_group();
          }
        }
      }
      if (failed) break;
    }
    if (lane == 0) bulk_wait_group<0>();                         // C is written before the kernel ends
    if (records) {
      trc[ag_trace::kAccWait] = t_acc;
      trc[ag_trace::kTiles] = n_tiles;
      trc[ag_trace::kTilesDone] = trc[ag_trace::kEnd] = globaltimer_ns();
    }
  }

  // ---------------- teardown ----------------
  if (__any_sync(0xffffffffu, failed)) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  cluster_sync_all();   // the peer may still read this CTA's smem / signal its barriers until here
  tcgen05_fence_after_thread_sync();
  if (warp == 1) tmem_dealloc_pair(tmem_base, kTmemCols);
}

}  // namespace wide
}  // namespace smr
