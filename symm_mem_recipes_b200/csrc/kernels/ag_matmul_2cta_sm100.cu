// The consumer GEMM of all_gather_matmul (upstream: `matmul_kernel_tma_persistent`,
// symm_mem_recipes/triton_all_gather_matmul.py:98-193, launched from :295-315)
// with tcgen05 `cta_group::2`: two CTAs on neighbouring SMs
// (a cluster of 2) share one 256 x BN tile.  Each CTA stages ITS OWN 128 rows
// of A and ITS OWN half of the B tile (BN/2 rows) with ordinary TMA loads — no
// cluster-multicast qualifier anywhere — and the leader CTA's single MMA thread
// issues `tcgen05.mma.cta_group::2`, which reads A and B from both CTAs'
// shared memory and writes each CTA's 128 accumulator rows into that CTA's own
// TMEM.  Per flop every SM pulls half as many B bytes out of L2 as a kernel with
// one CTA per 128 x BN tile would (ncu: tensor pipe 92 % active against 80 %).
//
// Hand-offs inside the pair:
//   full[s]        leader only.  The leader's producer arrives with the byte
//                  count of BOTH CTAs' loads; both CTAs' TMA loads complete on
//                  the leader's barrier (`.cta_group::2` form of the load).
//   empty[s]       both CTAs; `tcgen05.commit ... multicast::cluster` from the
//                  leader's MMA thread frees the stage in both.
//   tmem_full[b]   both CTAs; same multicast commit.
//   tmem_empty[b]  leader only, 8 arrivals: the four epilogue warps of each CTA
//                  (the peer's arrive through a shared::cluster address).
// Tail of the static schedule: when the last wave would fill only a few pairs
// (896 tiles on 74 pairs leave 8; a short prompt has fewer tiles than the GPU has
// pairs to begin with), each of its tiles is cut along K into 2 to 8 parts that run
// on as many pairs at once.  Every part stores its fp32
// partial accumulator to scratch memory (four columns x 128 rows contiguous, so
// that a warp's accesses are whole lines); a second kernel adds the parts up in their
// order, so the result does not depend on timing (merge_tail_kernel).  No CTA of a GEMM
// without a gather waits for another pair.
// The two 128-row blocks of a pair are two consecutive positions of the M
// schedule, not necessarily neighbours in memory: each CTA loads, waits for and
// stores its own block.
//
// Gather (mode 2, "push"): every rank broadcasts its own shard into the a_out of all
// ranks, with multimem.st through the NVSwitch from four ranks on, with plain peer
// stores below.  The shard is cut into pieces dealt to ALL GEMM CTAs, whose four
// epilogue warps push them in the time they would idle waiting for an accumulator,
// one round of tiles ahead of the first need; a block's arrival counter on every
// rank grows with each piece, and the TMA producer of a tile that reads a remote
// block waits (bounded) on the local counter.  Measured against the alternative of
// pulling the peers' shards with dedicated copier CTAs (a one-CTA-per-tile kernel
// this library used to carry): 1940 µs against 705-724 µs on 4 GPUs at the
// Llama-3-70B shape; an ordinary (non-symmetric) a_out is therefore served by this
// kernel through the internal symmetric buffer plus one local copy.
//
// Without a gather, and where there are whole waves of them, two tiles at a time are multiplied by matmul_wide.cuh.
#include "../device/pdl.cuh"
#include "../device/tcgen05_pair.cuh"
#include "ag_matmul_common.cuh"
#include "matmul_wide.cuh"
#include "residency.h"

namespace smr {

using namespace agmm;

namespace {

// Bytes of C that a tile has per row, and whether they leave through shared memory and TMA stores: in whole
// boxes of 128 bytes (a bf16 tile of 224 columns, or an fp8 tile of 192 or 224, would spill into its neighbour).
template <int BN, bool kFp8, bool kSwiGlu>
constexpr int pair_row_bytes() { return kFp8 ? BN : (kSwiGlu ? BN : 2 * BN); }
template <int BN, bool kFp8, bool kSwiGlu>
constexpr bool pair_tma_store() { return pair_row_bytes<BN, kFp8, kSwiGlu>() % 128 == 0; }

// kOut: the epilogue leaves through shared memory: each epilogue warp owns two 4 KB boxes (32 rows x 128
// bytes, 128-byte swizzle) that it fills from its accumulator rows and hands to a TMA store while it
// converts the next columns into the other box.  kBoxes > 2: a box for every 128 bytes of a tile's row, into which TMA
// brings the residual before the accumulator is complete.
template <int BN, int STAGES, bool kOut = false, int kBoxes = 2>
struct PairSmem {
  static constexpr uint32_t kABytes = kBM * kBK * 2;
  static constexpr uint32_t kBBytes = (BN / 2) * kBK * 2;     // this CTA's half of the B tile
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr uint32_t kRingBytes = kStageBytes * STAGES;
  static constexpr uint32_t kOutBoxBytes = 32 * 128;          // 32 rows x 64 bf16
  static constexpr uint32_t kOutOffset = kRingBytes;
  static constexpr uint32_t kOutBytes = kOut ? 4 * kBoxes * kOutBoxBytes : 0;
  static constexpr uint32_t kBarOffset = kRingBytes + kOutBytes;
  static constexpr uint32_t kNumBars = 2 * STAGES + 4 + 4 * kBoxes;   // the last ones: residual, [warp][box]
  static constexpr uint32_t kMiscOffset = kBarOffset + 8 * kNumBars;
  static constexpr uint32_t kTotal = kMiscOffset + 16 + 1024;
  static_assert(kStageBytes % 1024 == 0, "stage bases must stay 1024-byte aligned");
};

// kFp8: A, B, C (and the gathered A) hold e4m3 bytes.  All byte geometry stays
// (128-byte rows, 16 KB A stage, 32 bytes of K per MMA); a K block is then 128
// elements instead of 64 and the epilogue packs four outputs per 32-bit word.
// kSwiGlu (bf16, BN = 256): the rows of B are interleaved in groups of 128 so that every
// 256-column tile holds 128 gate columns followed by the 128 matching up columns;
// the epilogue writes SiLU(gate) * up, i.e. C is [M, N / 2] and tile ni covers its
// columns [128 ni, 128 ni + 128).  The activation never makes a round trip through
// memory and C is half as wide.  Since each CTA of a pair loads half of the tile's rows of
// B, gate and up rows may as well come from two separate halves of B (`b_pair`).
// kResidual (bf16, plain): C = bf16(bf16(A B^T) + residual), the residual add of a decoder layer without a pass of
// its own over C.
template <int BN, int STAGES, bool kFp8, bool kSwiGlu = false, bool kResidual = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
ag_matmul_2cta_kernel(const __grid_constant__ CUtensorMap tmap_a_shard,   // kResidual: the residual instead
                      const __grid_constant__ CUtensorMap tmap_a_out,
                      const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_c, const AgMatmulParams p) {
  constexpr bool kTmaStore = pair_tma_store<BN, kFp8, kSwiGlu>();
  static_assert(!kResidual || (kTmaStore && !kFp8 && !kSwiGlu), "the residual belongs to the plain bf16 epilogue");
  using L = PairSmem<BN, STAGES, kTmaStore, kResidual ? BN / 64 : 2>;
  extern __shared__ uint8_t smem_raw[];
  // same offset in both CTAs: the dynamic window starts at the same shared address
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kMiscOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  static_assert(!kSwiGlu || ((BN == 256 || BN == 224) && !kFp8), "the SwiGLU epilogue is built for bf16 tiles of 256 or 224 columns");

  uint32_t epoch = 0, flag_target = p.flag_target;
  if (p.mode == 2) {
    epoch = ld_relaxed_gpu(&p.header[0]) + 1u;
    flag_target = epoch * kArrivalUnits;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 8);   // 4 epilogue warps x 2 CTAs (used in the leader)
    }
    if constexpr (kResidual)
      for (int b = 0; b < 4 * (BN / 64); ++b) mbar_init(&bars[2 * STAGES + 4 + b], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a_shard);
    tma_prefetch_desc(&tmap_a_out);
    tma_prefetch_desc(&tmap_b);
    if constexpr (kTmaStore) tma_prefetch_desc(&tmap_c);
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
  const bool tr = p.trace != nullptr;
  uint64_t* trc = tr ? p.trace + (size_t)blockIdx.x * ag_trace::kTraceSlots : nullptr;
  if (tr && threadIdx.x == 0) trc[ag_trace::kStart] = globaltimer_ns();

  const int pair = (int)blockIdx.x >> 1;
  const int n_pairs = (int)gridDim.x >> 1;
  const int n_pair_rows = (p.n_blocks_m + 1) >> 1;         // 256-row tiles along M
  const int total_tiles = n_pair_rows * p.n_tiles_n;
  constexpr int kBKE = kFp8 ? 2 * kBK : kBK;                // elements of K per 128-byte row
  const int k_blocks = (p.K + kBKE - 1) / kBKE;
  const int rows_per_rank = p.blocks_per_rank * kBM;
  bool failed = false;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      PairWork w;
      uint64_t t_flag = 0, t_stage = 0, t_first = 0;
      bool first_remote = true;
      pdl_wait();
      for (int wi = 0; !failed && pair_work(p, pair, n_pairs, total_tiles, k_blocks, wi, w); ++wi) {
        const int t = w.tile;
        int prow, ni;
        tile_coords(p, n_pair_rows, t, prow, ni);
        const int mi = prow * 2 + (int)cta_rank;
        bool local = true;
        const CUtensorMap* amap = &tmap_a_out;
        int row0;
        if (mi < p.n_blocks_m) {
          const int mblk = scheduled_block(p, mi, local);
          row0 = mblk * kBM;
          if (p.mode != 0 && local) {
            amap = &tmap_a_shard;
            row0 -= p.rank * rows_per_rank;
          }
          if (!local) {
            const uint64_t t0 = tr ? globaltimer_ns() : 0;
            if (!wait_reached_acquire_sys(&p.flags[mblk], flag_target, p.timeout_ns)) {
              report_status(p.status, kTimeoutFlag, p.rank, blockIdx.x, mblk, kWhereGemmProgress);
              failed = true;
              break;
            }
            fence_proxy_async();
            if (tr) {
              const uint64_t dt = globaltimer_ns() - t0;
              t_flag += dt;
              if (first_remote) { t_first = dt; first_remote = false; }
            }
          }
        } else {
          row0 = p.n_blocks_m * kBM;   // odd tail: rows past M read as zero
        }
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_try_wait(&empty_bar[stage], phase ^ 1)) {
            const uint64_t t0 = tr ? globaltimer_ns() : 0;
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.timeout_ns)) {
              report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, stage, kWhereGemmEmpty);
              failed = true;
              break;
            }
            if (tr) t_stage += globaltimer_ns() - t0;
          }
          uint8_t* sa = smem + (size_t)stage * L::kStageBytes;
          uint8_t* sb = sa + L::kABytes;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2u * L::kStageBytes);
          const uint32_t full_leader = map_to_cta(smem_u32(&full_bar[stage]), 0);
          tma_load_2d_pair(sa, amap, full_leader, kb * kBKE, row0);
          tma_load_2d_pair(sb, &tmap_b, full_leader, kb * kBKE, ni * p.b_step + (int)cta_rank * p.b_pair);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (tr) {
        trc[ag_trace::kFlagWait] = t_flag;
        trc[ag_trace::kStageWait] = t_stage;
        trc[ag_trace::kFirstFlagWait] = t_first;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (leader && elect_one()) {
      constexpr uint32_t idesc = kFp8 ? umma_idesc_e4m3_f32(2 * kBM, BN) : umma_idesc_bf16_f32(2 * kBM, BN);
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      PairWork w;
      uint64_t t_tmem = 0, t_opnd = 0;
      for (int wi = 0; !failed && pair_work(p, pair, n_pairs, total_tiles, k_blocks, wi, w); ++wi) {
        if (!mbar_try_wait(&tmem_empty[acc], acc_phase ^ 1)) {
          const uint64_t t0 = tr ? globaltimer_ns() : 0;
          if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1, p.timeout_ns)) {
            report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, acc, kWhereGemmTmemEmpty);
            failed = true;
            break;
          }
          if (tr) t_tmem += globaltimer_ns() - t0;
        }
        tcgen05_fence_after_thread_sync();
        const uint32_t d_tmem = tmem_base + acc * 256u;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_try_wait(&full_bar[stage], phase)) {
            const uint64_t t0 = tr ? globaltimer_ns() : 0;
            if (!mbar_wait(&full_bar[stage], phase, p.timeout_ns)) {
              report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, stage, kWhereGemmFull);
              failed = true;
              break;
            }
            if (tr) t_opnd += globaltimer_ns() - t0;
          }
          tcgen05_fence_after_thread_sync();
          const uint32_t sa = smem_u32(smem + (size_t)stage * L::kStageBytes);
          const uint64_t da = umma_smem_desc_sw128(sa);
          const uint64_t db = umma_smem_desc_sw128(sa + L::kABytes);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            umma_ss_pair<kFp8>(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                               (kb != w.kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (failed) break;
        umma_commit_pair(&tmem_full[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
      if (tr) {
        trc[ag_trace::kTmemWait] = t_tmem;
        trc[ag_trace::kOperandWait] = t_opnd;
      }
    }
  } else {
    // ---------------- epilogue (warps 2..5 of both CTAs) ----------------
    const int quarter = warp & 3;
    uint32_t acc = 0, acc_phase = 0;
    const int etid = (int)threadIdx.x - 64;
    int next_piece = (int)blockIdx.x, round = 0;
    const int all_pieces = p.blocks_per_rank * p.pieces;
    pdl_wait();
    [[maybe_unused]] int out_box = 0;                  // which of this warp's two output boxes is filled next
    // Residual: a tile's boxes are brought in while the tile is multiplied; res_phase has the parity of each box's barrier.
    // (Loaded by the lanes themselves, 16 bytes of 32 rows at a time, it cost 16384 x 8192 x 3584 123 us on top of 624.)
    [[maybe_unused]] uint64_t* res_full = bars + 2 * STAGES + 4 + quarter * (BN / 64);
    [[maybe_unused]] uint32_t res_phase = 0;
    if (p.mode == 2 && !push_entry_barrier(p, (int)blockIdx.x, etid)) failed = true;
    const bool trt = tr && etid == 0;
    uint64_t t_push = 0, t_acc = 0, n_units = 0;
    if (trt) trc[ag_trace::kEntered] = globaltimer_ns();
    PairWork w;
    for (int wi = 0; !failed && pair_work(p, pair, n_pairs, total_tiles, k_blocks, wi, w); ++wi) {
      const int t = w.tile;
      int prow, ni;
      tile_coords(p, n_pair_rows, t, prow, ni);
      const int mi = prow * 2 + (int)cta_rank;
      bool local_unused;
      const bool valid = mi < p.n_blocks_m;
      const int mblk = valid ? scheduled_block(p, mi, local_unused) : 0;
      if (p.mode == 2) {
        const uint64_t t0 = trt ? globaltimer_ns() : 0;
        next_piece = push_pieces(p, next_piece, (int)gridDim.x,
                                 pieces_due(p, round, n_pairs, 2, all_pieces), etid);
        ++round;
        if (trt) t_push += globaltimer_ns() - t0;
      }
      if constexpr (kResidual) {
        if (w.part < 0 && valid && mblk * kBM + quarter * 32 < p.M && lane == 0) {
          bulk_wait_group_read<0>();                   // the stores of the tile before have read these boxes
          for (int c = 0; c < BN / 64 && ni * BN + c * 64 < p.N; ++c) {
            mbar_arrive_expect_tx(&res_full[c], L::kOutBoxBytes);
            tma_load_2d(smem + L::kOutOffset + ((size_t)quarter * (BN / 64) + c) * L::kOutBoxBytes, &tmap_a_shard, &res_full[c],
                        ni * BN + c * 64, mblk * kBM + quarter * 32);
          }
        }
      }
      {
        const uint64_t t0 = trt ? globaltimer_ns() : 0;
        if (!mbar_wait(&tmem_full[acc], acc_phase, p.timeout_ns)) {
          if (lane == 0)
            report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, acc, kWhereGemmTmemFull);
          failed = true;
          break;
        }
        if (trt) { t_acc += globaltimer_ns() - t0; ++n_units; }
      }
      tcgen05_fence_after_thread_sync();
      const int row = mblk * kBM + quarter * 32 + lane;
      const bool row_ok = valid && row < p.M;
      const uint32_t taddr = tmem_base + acc * 256u + ((uint32_t)(quarter * 32) << 16);
      auto release_accumulator = [&]() {
        tcgen05_fence_before_thread_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));
      };
      constexpr int kOutCols = kSwiGlu ? BN / 2 : BN;                // columns of C in this tile
      const int n_out = kSwiGlu ? p.N >> 1 : p.N;                    // columns of C
      const int col0 = ni * kOutCols;
      uint8_t* crow = reinterpret_cast<uint8_t*>(p.c) + ((size_t)row * n_out + col0) * (kFp8 ? 1 : 2);
      if (w.part >= 0) {
        // ---- split-K tail: park the fp32 partial for merge_tail_kernel ----
        const size_t blk = (size_t)kBM * BN;                         // floats per CTA block
        const int r = quarter * 32 + lane;
        float* mine = p.tail_scratch + (((size_t)w.tail_idx * p.tail_splits + w.part) * 2 + cta_rank) * blk + r * 4;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
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
      } else if constexpr (kTmaStore) {
        // One box (128 bytes of every row) at a time: accumulator columns -> packed words -> this warp's free
        // box (16-byte chunk j of row r sits at chunk j ^ (r & 7): the 128-byte swizzle of the tensor map,
        // conflict-free for the warp's stores) -> one TMA store.
        constexpr int kBoxes = pair_row_bytes<BN, kFp8, kSwiGlu>() / 128;
        constexpr int kBoxCols = kOutCols / kBoxes;                  // columns of C per box
        const uint32_t box0 = smem_u32(smem + L::kOutOffset) + (uint32_t)quarter * (kResidual ? kBoxes : 2) * L::kOutBoxBytes;
        const bool store_ok = valid && mblk * kBM + quarter * 32 < p.M;
#pragma unroll 1
        for (int c = 0; c < kBoxes; ++c) {
          // 64 accumulator columns in flight: the whole box, or half of it where two go into one of C's bytes (fp8)
          // or columns (SwiGLU)
          constexpr int kPasses = kFp8 || kSwiGlu ? 2 : 1;
          if constexpr (kResidual) out_box = c;
          const uint32_t box = box0 + (uint32_t)out_box * L::kOutBoxBytes;
          const uint32_t rowaddr = box + (uint32_t)lane * 128u;
          const uint32_t sw = (uint32_t)(lane & 7);
#pragma unroll
          for (int h = 0; h < kPasses; ++h) {
            uint32_t v[2][32];
            if constexpr (kSwiGlu) {
              tmem_ld_32x32b_x32(taddr + (uint32_t)(c * 64 + h * 32), v[0]);             // gate columns
              tmem_ld_32x32b_x32(taddr + (uint32_t)(BN / 2 + c * 64 + h * 32), v[1]);    // the matching up columns
            } else {
              tmem_ld_32x32b_x32(taddr + (uint32_t)(c * kBoxCols + h * 64), v[0]);
              tmem_ld_32x32b_x32(taddr + (uint32_t)(c * kBoxCols + h * 64 + 32), v[1]);
            }
            if constexpr (kResidual) {
              if (store_ok && col0 + c * kBoxCols < n_out) {
                if (!mbar_wait(&res_full[c], (res_phase >> c) & 1u, p.timeout_ns)) {
                  if (lane == 0) report_status(p.status, kTimeoutMbarrier, p.rank, blockIdx.x, c, kWhereGemmFull);
                  failed = true;
                }
                res_phase ^= 1u << c;
              }
            } else if (h == 0) {
              if (lane == 0) bulk_wait_group_read<1>();      // the store that last read this box is done with it
              __syncwarp();
            }
            tmem_ld_wait();
            // the accumulator is in registers: hand it back before the stores
            if (c == kBoxes - 1 && h == kPasses - 1) release_accumulator();
#pragma unroll
            for (int j = 0; j < 8 / kPasses; ++j) {
              Vec16 o;
              if constexpr (kFp8) {
                const uint32_t* q = v[j / 2] + (j & 1) * 16;
                auto f = [q](int i) { return __uint_as_float(q[i]); };
                o.x = pack_e4m3x4(f(0), f(1), f(2), f(3)); o.y = pack_e4m3x4(f(4), f(5), f(6), f(7));
                o.z = pack_e4m3x4(f(8), f(9), f(10), f(11)); o.w = pack_e4m3x4(f(12), f(13), f(14), f(15));
              } else {
                const uint32_t* q = v[kSwiGlu ? 0 : j / 4] + (j & 3) * 8;
                float y[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  y[i] = __uint_as_float(q[i]);
                  if constexpr (kSwiGlu) y[i] = y[i] / (1.0f + __expf(-y[i])) * __uint_as_float(v[1][j * 8 + i]);
                }
                o.x = pack_bf16x2(y[0], y[1]); o.y = pack_bf16x2(y[2], y[3]);
                o.z = pack_bf16x2(y[4], y[5]); o.w = pack_bf16x2(y[6], y[7]);
              }
              const uint32_t chunk = rowaddr + (((uint32_t)(h * (8 / kPasses) + j) ^ sw) << 4);
              if constexpr (kResidual) o = add_bf16x8(o, ld_shared_16(chunk));
              st_shared_16(chunk, o.x, o.y, o.z, o.w);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (store_ok && col0 + c * kBoxCols < n_out) {
              uint8_t* src = smem + L::kOutOffset + ((size_t)quarter * (kResidual ? kBoxes : 2) + out_box) * L::kOutBoxBytes;
              tma_store_2d(&tmap_c, src, col0 + c * kBoxCols, mblk * kBM + quarter * 32);
            }
            bulk_commit_group();
          }
          if constexpr (!kResidual) out_box ^= 1;
        }
      } else if constexpr (kSwiGlu) {
#pragma unroll 1
        for (int c = 0; c < kOutCols / 16; ++c) {
          uint32_t g[16], u[16];
          tmem_ld_32x32b_x16(taddr + (uint32_t)(c * 16), g);
          tmem_ld_32x32b_x16(taddr + (uint32_t)(BN / 2 + c * 16), u);
          tmem_ld_wait();
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            if (row_ok && col0 + c * 16 + v * 8 < n_out) {
              float y[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float x = __uint_as_float(g[v * 8 + i]);
                y[i] = x / (1.0f + __expf(-x)) * __uint_as_float(u[v * 8 + i]);
              }
              st_16(crow + (c * 16 + v * 8) * 2, Vec16{pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]),
                                                       pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7])});
            }
          }
        }
        release_accumulator();
      } else {
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + (uint32_t)(c * 32), r);
          tmem_ld_wait();
          if constexpr (kFp8) {
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              if (row_ok && col0 + c * 32 + v * 16 < p.N) {
                auto f = [&r, v](int i) { return __uint_as_float(r[v * 16 + i]); };
                Vec16 o;
                o.x = pack_e4m3x4(f(0), f(1), f(2), f(3)); o.y = pack_e4m3x4(f(4), f(5), f(6), f(7));
                o.z = pack_e4m3x4(f(8), f(9), f(10), f(11)); o.w = pack_e4m3x4(f(12), f(13), f(14), f(15));
                st_16(crow + c * 32 + v * 16, o);
              }
            }
          } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              if (row_ok && col0 + c * 32 + v * 8 < p.N) {
                Vec16 o;
                o.x = pack_bf16x2(__uint_as_float(r[v * 8 + 0]), __uint_as_float(r[v * 8 + 1]));
                o.y = pack_bf16x2(__uint_as_float(r[v * 8 + 2]), __uint_as_float(r[v * 8 + 3]));
                o.z = pack_bf16x2(__uint_as_float(r[v * 8 + 4]), __uint_as_float(r[v * 8 + 5]));
                o.w = pack_bf16x2(__uint_as_float(r[v * 8 + 6]), __uint_as_float(r[v * 8 + 7]));
                st_16(crow + (c * 32 + v * 8) * 2, o);
              }
            }
          }
        }
        release_accumulator();
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if constexpr (kTmaStore) {
      if (lane == 0) bulk_wait_group<0>();             // C is written before the kernel ends
    }
    if (trt) trc[ag_trace::kTilesDone] = globaltimer_ns();
    if (p.mode == 2 && !failed) {
      const uint64_t t0 = trt ? globaltimer_ns() : 0;
      push_pieces(p, next_piece, (int)gridDim.x, all_pieces, etid);
      if (trt) t_push += globaltimer_ns() - t0;
    }
    if (trt) {
      trc[ag_trace::kPush] = t_push;
      trc[ag_trace::kAccWait] = t_acc;
      trc[ag_trace::kTiles] = n_units;
      trc[ag_trace::kEnd] = globaltimer_ns();
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
  if (p.mode == 2 && threadIdx.x == 0) {
    uint32_t done = atomicAdd(&p.header[1], 1u);
    if (done == gridDim.x - 1) {
      p.header[1] = 0u;
      __threadfence();
      st_release_gpu(&p.header[0], epoch);
    }
  }
}

// The parts of the tail's tiles added up in their order, with the GEMM's three ends.  A warp takes eight rows of four
// groups of eight columns: its loads are whole lines of the scratch layout, its stores 64 bytes of a row.  Bound by the
// pass through L2; launched under the GEMM (its CTAs fit beside the GEMM's), it begins when the last part is stored.
// A kernel of its own, because parts that wait for one another inside the GEMM need all of its CTAs resident at once:
// against waits without that guarantee 1024 x 1280 x 8192 27.0 -> 25.0 us, 200 x 512 x 8192 11.8 -> 10.6, 200 x 1280 x
// 4096 11.3 -> 11.6; a cooperative launch, which gives the guarantee, took fp8 4096 x 3584 x 8192 from 103.2 to 106.2.
constexpr int kMergeThreads = 256;
template <int BN, bool kFp8, bool kSwiGlu, bool kResidual>
__global__ void __launch_bounds__(kMergeThreads) merge_tail_kernel(const AgMatmulParams p) {
  pdl_launch_dependents();
  constexpr int kOutCols = kSwiGlu ? BN / 2 : BN, kGroupBlocks = kOutCols / 32, kBlk = kBM * BN;
  const int lane = threadIdx.x & 31;
  int u = (int)(blockIdx.x * (kMergeThreads / 32) + (threadIdx.x >> 5));
  const int g = u % kGroupBlocks * 4 + (lane >> 3);                  // columns 8 g .. 8 g + 7 of the tile's C
  u /= kGroupBlocks;
  const int r = u % (kBM / 8) * 8 + (lane & 7);                      // row of the CTA's block
  u /= kBM / 8;
  const int cta = u & 1, tail_idx = u >> 1;
  if (tail_idx >= p.tail_tiles) return;
  const int n_pair_rows = (p.n_blocks_m + 1) >> 1;
  int prow, ni;
  work_coords(p, n_pair_rows, n_pair_rows * p.n_tiles_n - 2 * p.wide_units - p.tail_tiles + tail_idx, 1, prow, ni);
  const int mi = prow * 2 + cta, n_out = kSwiGlu ? p.N >> 1 : p.N, col = ni * kOutCols + g * 8;
  if (mi >= p.n_blocks_m || col >= n_out) return;
  bool local_unused;
  const int row = scheduled_block(p, mi, local_unused) * kBM + r;
  if (row >= p.M) return;
  const float* src = p.tail_scratch + ((size_t)tail_idx * p.tail_splits * 2 + cta) * kBlk + (size_t)g * (2 * kBM * 4) + r * 4;
  const size_t up = (size_t)(BN / 8) * (kBM * 4);                    // from a gate column to the matching up column
  pdl_wait();
  constexpr int kHalves = kSwiGlu ? 2 : 1, kInFlight = 4;            // parts whose loads are in flight at once
  float s[kHalves][8] = {};
  for (int i0 = 0; i0 < p.tail_splits; i0 += kInFlight) {
    Vec16 v[kInFlight][kHalves][2];
#pragma unroll
    for (int i = 0; i < kInFlight; ++i)
#pragma unroll
      for (int h = 0; h < kHalves; ++h)
        if (i0 + i < p.tail_splits) {
          const float* q = src + (size_t)(i0 + i) * 2 * kBlk + h * up;
          v[i][h][0] = ld_16_stream(q);
          v[i][h][1] = ld_16_stream(q + kBM * 4);
        }
#pragma unroll
    for (int i = 0; i < kInFlight; ++i)                              // in part order
#pragma unroll
      for (int h = 0; h < kHalves; ++h)
        if (i0 + i < p.tail_splits) {
          const Vec16 &a = v[i][h][0], &b = v[i][h][1];
          s[h][0] += __uint_as_float(a.x); s[h][1] += __uint_as_float(a.y);
          s[h][2] += __uint_as_float(a.z); s[h][3] += __uint_as_float(a.w);
          s[h][4] += __uint_as_float(b.x); s[h][5] += __uint_as_float(b.y);
          s[h][6] += __uint_as_float(b.z); s[h][7] += __uint_as_float(b.w);
        }
  }
  if constexpr (kSwiGlu) {
#pragma unroll
    for (int q = 0; q < 8; ++q) s[0][q] = s[0][q] / (1.0f + __expf(-s[0][q])) * s[1][q];
  }
  const size_t at = (size_t)row * n_out + col;
  if constexpr (kFp8) {
    st_8(reinterpret_cast<uint8_t*>(p.c) + at, pack_e4m3x4(s[0][0], s[0][1], s[0][2], s[0][3]),
         pack_e4m3x4(s[0][4], s[0][5], s[0][6], s[0][7]));
  } else {
    Vec16 o;
    o.x = pack_bf16x2(s[0][0], s[0][1]); o.y = pack_bf16x2(s[0][2], s[0][3]);
    o.z = pack_bf16x2(s[0][4], s[0][5]); o.w = pack_bf16x2(s[0][6], s[0][7]);
    if constexpr (kResidual) o = add_bf16x8(o, ld_16(p.residual + at));
    st_16(p.c + at, o);
  }
}

cudaLaunchConfig_t overlapped(int grid, int threads, uint32_t smem, bool overlap, cudaLaunchAttribute (&attr)[1],
                              cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cfg;
}

template <int BN, bool kFp8, bool kSwiGlu, bool kResidual>
int launch_merge(const AgMatmulParams& p, cudaStream_t stream) {
  constexpr int kWarpsPerBlock = kBM / 8 * (kSwiGlu ? BN / 2 : BN) / 32;
  const int warps = p.tail_tiles * 2 * kWarpsPerBlock;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = overlapped((warps + kMergeThreads / 32 - 1) / (kMergeThreads / 32), kMergeThreads, 0, true, attr, stream);
  return (int)cudaLaunchKernelEx(&cfg, merge_tail_kernel<BN, kFp8, kSwiGlu, kResidual>, p);
}

template <int BN, int STAGES, bool kFp8, bool kSwiGlu = false, bool kResidual = false>
int launch_pair_variant(const CUtensorMap& ta_shard, const CUtensorMap& ta_out, const CUtensorMap& tb,
                        const CUtensorMap& tc, const AgMatmulParams& p, int grid, bool overlap, cudaStream_t stream) {
  using L = PairSmem<BN, STAGES, pair_tma_store<BN, kFp8, kSwiGlu>(), kResidual ? BN / 64 : 2>;
  static_assert(L::kTotal <= 232448, "shared memory limit exceeded");
  auto kern = ag_matmul_2cta_kernel<BN, STAGES, kFp8, kSwiGlu, kResidual>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kTotal);
  if (e != cudaSuccess) return (int)e;
  // The pairs of a gather wait for one another's pieces: all of them must be resident.
  if (p.mode != 0)
    if (int rc = check_co_resident(kern, grid, kGemmThreads, L::kTotal, 2)) return rc;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = overlapped(grid, kGemmThreads, L::kTotal, overlap, attr, stream);
  e = cudaLaunchKernelEx(&cfg, kern, ta_shard, ta_out, tb, tc, p);
  if (e != cudaSuccess || p.tail_tiles == 0) return (int)e;
  if constexpr (kSwiGlu && BN == 224) return cudaErrorInvalidValue;  // never cut: its columns are no whole groups of the merge
  else return launch_merge<BN, kFp8, kSwiGlu, kResidual>(p, stream);
}

template <bool kSwiGlu, bool kResidual>
int launch_wide(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tr,
                const AgMatmulParams& p, int grid, bool overlap, cudaStream_t stream) {
  auto kern = p.trace != nullptr ? wide::matmul_wide_kernel<kSwiGlu, kResidual, true> : wide::matmul_wide_kernel<kSwiGlu, kResidual, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wide::kSmemBytes);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = overlapped(grid, wide::kThreads, wide::kSmemBytes, overlap, attr, stream);
  e = cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, tr, p);
  if (e != cudaSuccess || p.tail_tiles == 0) return (int)e;
  return launch_merge<wide::kBN, false, kSwiGlu, kResidual>(p, stream);
}

}  // namespace

namespace {

// Parts a tile of the tail is cut into: `rem` tiles in the last wave of `pairs` pairs.
int tail_parts(int rem, int pairs, int k_blocks, int most) {
  if (rem <= 0 || rem * 2 > pairs) return 1;
  int splits = pairs / rem;
  if (splits > kMaxTailParts) splits = kMaxTailParts;
  if (most > 0 && splits > most) splits = most;
  while (splits > 1 && k_blocks < 2 * splits) --splits;
  return splits;
}

size_t tail_scratch_bytes(int tiles, int parts, int bn) { return (size_t)tiles * parts * 2 * kBM * bn * sizeof(float); }

// Units of two tiles (matmul_wide.cuh) that a GEMM of `rows` x `cols` tiles of 256 x 256 is multiplied in: as many whole
// waves of them as there are, the rest one tile at a time.  bf16 only: in fp8 the same loads feed twice the flops, and
// 4096 and 16384 x 3584 x 8192 take 95 and 362 us either way.  The end of a unit costs about 4000 cycles more than that
// of two single tiles (both accumulators have to be read before the next unit), so K has to be long.  Loops of calls at
// 1000 W, all in one session, in turn: us (median SM clock, MHz) one tile at a time / two:
//     16384 x 8192 x 1024    218 (1166) / 224 (1485)      16384 x 3584 x 8192    748 (1162) / 701 (1327)
//     16384 x 8192 x 2048    404 (1297) / 410 (1402)       4096 x 7168 x 8192    377 (1237) / 359 (1342)
//     16384 x 4096 x 4096    399 (1297) / 401 (1365)      16384 x 4096 x 6144    634 (1181) / 605 (1327)
//   with SwiGLU (columns of C)
//      9000 x 8192 x 4096    889 (1275) / 915 (1357)       2048 x 7168 x 8192    383 (1162) / 366 (1327)
//                                                         32768 x 7168 x 8192   5830 (1095) / 5657 (1282)
//   with residual (one stage less one tile at a time)
//     16384 x 8192 x 2048    441 (1162) / 466 (1327)      32768 x 8192 x 3584   1617 (1027) / 1578 (1271)
//                                                         16384 x 8192 x 7168   1539 (1087) / 1453 (1286)
// An odd column of tiles comes after all units and reads all of A again:
//      8192 x 1280 x 8192 (5 columns)  140 / 140          32768 x 1280 x 8192 (5)  530 / 549
//     32768 x 1792 x 8192 (7)          736 / 740          32768 x 2304 x 8192 (9)  941 / 935
// Single calls at a high clock (4 ms of pause before each, L2 cold), where power does not limit, lose nothing: 2048 x 5120
// x 8192 118 / 118, 4096 x 3584 x 8192 159 / 159, 2048 x 8192 x 5120 120 / 119, 1024 x 7168 x 8192 with SwiGLU 165 / 161, with
// residual 1280 x 8192 x 3584 71 / 69 and 2048 x 8192 x 3584 99 / 95, 16384 x 3584 x 8192 605 / 585.
int plan_wide_units(int rows, int cols, int pairs, int K, int elem_bytes, bool residual) {
  if (elem_bytes != 2 || K < (residual ? 3072 : 5120) || (cols % 2 != 0 && cols < 9)) return 0;
  return rows * (cols / 2) / pairs * pairs;
}

}  // namespace

// Tile width and tail of a GEMM by a model of its time, fitted to loops of calls (so at the clocks the power limit leaves)
// of every width on 35 bf16 and 28 fp8 shapes (M 131 to 32768): a wave of n of the P pairs takes, per K block of 128
// bytes, t1 with few pairs at work (the tensor core's own rate) up to t1 + t2 with all of them (shared L2 and power),
// so narrow tiles win where tiles are few and 256 columns where waves are full; cutting the last wave along K costs 2 us
// and a pass of the parts through L2 (509 x 1280 x 8192: 128 columns in 3 parts are 2 us faster than 256 in 7).  Rows
// whose pitch is no multiple of 128 bytes make every TMA row touch two L2 lines: `skew` more per K block.  A tile
// cannot take less than its epilogue, `epi`, where K is short (244 x 1024 x 640: 6.6 us at 128 columns, 7.5 at 192).
// Where there are units of two tiles and K is 5120 or more, whole waves are priced at 0.94.  All of them, not only those of
// units: that choice differs in 33 of 120000 random shapes, half of which are faster either way (9750 x 1312 x 5280 124 us, with
// only the units' waves 116; 16363 x 1296 x 9304 372, 428).  The shorter K that units with a residual take is priced at 1: they save 2 to 3 %
// there, less than 192 columns do where those fill the waves (1240 x 8192 x 3584 66.5 us, 256 columns 69.6).  On the shapes of
// the fit and ten more the width that the plan picks is on average 0.1 % slower than the best one, at worst 3.8 % (148 x 1856 x
// 7008: 13.2 us at 192 columns in parts, 12.7 at 128; then 2992 x 6224 x 704 with 1.6 %: 26.9 at 192, 26.5 at 256).
// Examples, fp8, with the figures of before (fitted in short bursts) and now: 4096 x 3584 x 8192 103 -> 97 us (192 -> 256
// columns), 16384 x 3584 x 8192 386 -> 362, 1024 x 8192 x 8192 65 -> 61; bf16 2992 x 6224 x 704 29.4 -> 27.6.
MatmulPlan plan_matmul(int M, int N, int K, int elem_bytes, int epilogue, int block_n, int num_sms, int max_splits, bool residual) {
  struct Width { int bn; double t1, t2, skew, epi; };               // microseconds
  constexpr Width kBf16[] = {{256, 0.29, 0.15, 0.03, 3.2}, {192, 0.218, 0.135, 0.03, 2.6}, {128, 0.135, 0.12, 0.04, 2.3}};
  constexpr Width kFp8[] = {{256, 0.29, 0.135, 0.04, 2.7}, {192, 0.225, 0.13, 0.065, 3.0}, {128, 0.125, 0.13, 0.08, 2.0}};
  const Width(&widths)[3] = elem_bytes == 1 ? kFp8 : kBf16;
  const int pairs = num_sms < 4 ? 1 : num_sms / 2, rows = (M + 2 * kBM - 1) / (2 * kBM);
  const int k_blocks = (K * elem_bytes + 127) / 128;
  MatmulPlan best{block_n != 0 ? block_n : 256, 1, 0, 0};
  double best_cost = -1;
  for (const Width& w : widths) {
    // a width the caller (or the SwiGLU epilogue) asks for is taken with the figures of the nearest one
    if (block_n != 0 || epilogue != 0) {
      if (w.bn != (block_n == 128 || block_n == 192 ? block_n : 256)) continue;
    }
    const int bn = block_n != 0 ? block_n : w.bn;
    const int tiles = rows * (epilogue != 0 ? (N / 2 + bn / 2 - 1) / (bn / 2) : (N + bn - 1) / bn);
    const double t1 = w.t1 + (K * elem_bytes % 128 != 0 ? w.skew : 0.0);
    auto wave_us = [&](int n, int parts) {
      const double us = k_blocks * (t1 + w.t2 * n * parts / pairs) / parts;
      return us > w.epi ? us : w.epi;
    };
    const int rem = tiles % pairs;
    const int wide_units = bn == 256 ? plan_wide_units(rows, tiles / rows, pairs, K, elem_bytes, residual) : 0;
    double cost = tiles / pairs * wave_us(pairs, 1) * (wide_units > 0 && K >= 5120 ? 0.94 : 1.0);
    int parts = 1;
    if (rem > 0) {
      double tail = wave_us(rem, 1);
      for (int most = tail_parts(rem, pairs, k_blocks, max_splits < 0 ? -max_splits : max_splits); most >= 2; --most) {
        const double cut = wave_us(rem, most) + 2.0 + 0.25e-6 * tail_scratch_bytes(rem, most, bn);
        if (cut < tail || max_splits < 0) { tail = cut; parts = most; }
        if (max_splits < 0) break;
      }
      cost += tail;
    }
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best.block_n = bn;
      best.tail_splits = parts;
      best.tail_bytes = parts > 1 ? tail_scratch_bytes(rem, parts, bn) : 0;
      best.wide_units = wide_units;
    }
  }
  // Gate and up in two halves of B: 112 columns of each, uncut, where that fills the pairs better (K 8192, us): 300 x 7168
  // 50 -> 45, 509 x 7168 57 -> 53 (64 tiles on 74 pairs instead of 56), 509 x 14336 106 -> 103, 900 x 7168 113 -> 107, 1500 x
  // 7168 150 -> 146; 385 x 4000 x 2048 24.5 -> 21.1.  Its rows of C are 224 bytes, so the lanes store them themselves.
  if (epilogue == 2 && block_n == 0 && max_splits >= 0) {
    const int tiles = rows * ((N / 2 + 111) / 112), rem = tiles % pairs;
    auto wave_us = [&](int n) {
      const double us = k_blocks * (0.254 + (K % kBK != 0 ? 0.03 : 0.0) + 0.143 * n / pairs);
      return us > 4.0 ? us : 4.0;
    };
    if (tiles / pairs * wave_us(pairs) + (rem > 0 ? wave_us(rem) : 0.0) < 0.97 * best_cost) best = MatmulPlan{224, 1, 0, 0};
  }
  return best;
}

int gemm_kernels(int M, int N, int K, int elem_bytes, int num_sms, bool gather) {
  if (!gather) return plan_matmul(M, N, K, elem_bytes, 0, 0, num_sms, 0, false).tail_splits > 1 ? 2 : 1;
  const int tiles = (M + 2 * kBM - 1) / (2 * kBM) * ((N + 255) / 256), pairs = num_sms < 4 ? 1 : num_sms / 2;
  return tail_parts(tiles % pairs, pairs, (K * elem_bytes + 127) / 128, 0) > 1 ? 2 : 1;
}

int launch_ag_matmul_2cta(const AgMatmulArgs& a, cudaStream_t stream) {
  if (a.elem_bytes != 0 && a.elem_bytes != 1 && a.elem_bytes != 2) return cudaErrorInvalidValue;
  const bool fp8 = a.elem_bytes == 1;
  const int es = fp8 ? 1 : 2;
  const int align = 16 / es;                                       // elements per 16 bytes
  if (a.N % align != 0 || a.K % align != 0 || a.M <= 0 || a.N <= 0 || a.K <= 0) return cudaErrorInvalidValue;
  if (a.mode != 0 && a.mode != 2) return cudaErrorInvalidValue;
  const bool comm = a.mode == 2;
  if (comm) {
    if (a.world_size < 2 || a.rows_per_rank % kBM != 0 || a.rows_per_rank * a.world_size != a.M ||
        a.a_out == nullptr || a.pads == nullptr || a.aout_buffers == nullptr || a.local_pad == nullptr)
      return cudaErrorInvalidValue;
    if ((uint32_t)(a.M / kBM) + 2u > kFusedFlagSlots) return cudaErrorInvalidValue;
  }
  const int bn = a.block_n;
  if (bn != 128 && bn != 192 && bn != 224 && bn != 256) return cudaErrorInvalidValue;
  const bool swiglu = a.epilogue != 0;
  if (a.epilogue < 0 || a.epilogue > 2) return cudaErrorInvalidValue;
  // bf16, 256-column tiles, or 224 uncut; interleaved in groups of 128 rows of B: whole groups of 256 columns only
  if (swiglu && (fp8 || (bn != 256 && (bn != 224 || a.epilogue != 2 || a.tail_scratch != nullptr || comm)) ||
                 a.N % (a.epilogue == 1 ? 256 : 16) != 0))
    return cudaErrorInvalidValue;
  if (a.residual != nullptr && (swiglu || fp8 || comm || bn == 224 || (uintptr_t)a.residual % 16 != 0))
    return cudaErrorInvalidValue;

  AgMatmulParams p{};
  p.c = static_cast<__nv_bfloat16*>(a.c);
  p.M = a.M; p.N = a.N; p.K = a.K;
  p.elem_bytes = es;
  // with the SwiGLU epilogue a tile is 128 columns of C, whichever way its gate and up rows are stored
  p.n_tiles_n = swiglu ? (a.N / 2 + bn / 2 - 1) / (bn / 2) : (a.N + bn - 1) / bn;
  p.b_step = a.epilogue == 2 ? bn / 2 : bn;
  p.b_pair = a.epilogue == 2 ? a.N / 2 : bn / 2;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual);
  p.panel_w = a.panel_w > 0 ? (a.panel_w < p.n_tiles_n ? a.panel_w : p.n_tiles_n)
                            : pick_panel_w(p.n_tiles_n, (size_t)bn * a.K * es);
  p.n_blocks_m = (a.M + kBM - 1) / kBM;
  p.rank = comm ? a.rank : 0;
  p.world_size = comm ? a.world_size : 1;
  p.blocks_per_rank = comm ? a.rows_per_rank / kBM : p.n_blocks_m;
  p.mode = a.mode;
  p.lead = 0;
  p.pieces = 1;
  if (comm) {
    p.lead = p.blocks_per_rank < 4 ? p.blocks_per_rank : 4;
    if (a.lead >= 0) p.lead = a.lead < p.blocks_per_rank ? a.lead : p.blocks_per_rank;
    p.push_ahead = a.push_ahead > 0 ? a.push_ahead : 1;
    size_t block_vecs = (size_t)kBM * a.K * es / 16;
    p.pieces = block_vecs >= 8192 ? 16 : (block_vecs >= 1024 ? 4 : 1);
    // A CTA's epilogue warps take 40-60 µs to broadcast 128 KB, about one round of tiles, which is all the
    // lead the schedule gives a piece once the own blocks are used up: with eight ranks (16 blocks per rank,
    // 1.7 pieces of 128 KB per CTA) the CTAs waited 165 µs per call for remote blocks.  So the smaller the
    // shard, the finer the pieces: about six per CTA over the whole shard (64 per block at eight ranks of
    // the headline shape, 32 at four, 16 at two; on four ranks 64 measured 10-29 µs faster than 16).
    while (p.pieces < 256 && (size_t)p.blocks_per_rank * p.pieces < (size_t)6 * a.num_sms &&
           (size_t)(2 * p.pieces) * 128 <= block_vecs)
      p.pieces *= 2;
    if (a.push_pieces > 0) {
      if ((a.push_pieces & (a.push_pieces - 1)) != 0 || (uint32_t)a.push_pieces > kArrivalUnits) return cudaErrorInvalidValue;
      p.pieces = a.push_pieces;
      while (p.pieces > 1 && (size_t)p.pieces * 128 > block_vecs) p.pieces >>= 1;   // a piece feeds 128 threads at least once
    }
  }
  p.flags = comm ? a.local_pad + kFlagSlotsBase + 2 : nullptr;
  p.flag_target = 1u;
  p.header = comm ? a.local_pad + kFlagSlotsBase : nullptr;
  p.a_local = static_cast<const char*>(a.a_local);
  p.aout_buffers = a.aout_buffers;
  p.aout_mc = a.push_plain_stores ? nullptr : a.aout_mc;
  p.aout_offset = a.aout_offset;
  p.a_out = static_cast<char*>(a.a_out);
  p.pads = a.pads;
  p.barrier_block_base = a.barrier_block_base;
  p.timeout_ns = a.timeout_ns;
  p.status = a.status;
  p.trace = a.trace;

  CUtensorMap ta_shard, ta_out, tb, tc;
  int rows_local = comm ? a.rows_per_rank : a.M;
  // without a gather nobody reads the shard's map, and the residual (32 x 64 boxes, as C) takes its place
  if (a.residual != nullptr ? make_tmap(&ta_shard, a.residual, (uint64_t)a.M, (uint64_t)a.N, 32, es)
                            : make_tmap(&ta_shard, a.a_local, (uint64_t)rows_local, (uint64_t)a.K, kBM, es))
    return cudaErrorInvalidValue;
  if (make_tmap(&ta_out, comm ? a.a_out : a.a_local, (uint64_t)a.M, (uint64_t)a.K, kBM, es))
    return cudaErrorInvalidValue;
  if (make_tmap(&tb, a.b, (uint64_t)a.N, (uint64_t)a.K, (uint32_t)(bn / 2), es)) return cudaErrorInvalidValue;
  // C as the TMA stores of the plain bf16 epilogue see it: boxes of 32 rows x 64 columns
  const int c_cols = swiglu ? a.N / 2 : a.N;
  if (make_tmap(&tc, a.c, (uint64_t)a.M, (uint64_t)c_cols, 32, es)) return cudaErrorInvalidValue;

  const int total_tiles = ((p.n_blocks_m + 1) / 2) * p.n_tiles_n;
  const int max_pairs = a.num_sms / 2;
  if (max_pairs < 1) return cudaErrorInvalidValue;
  const int k_blocks = (a.K * es + 127) / 128;                    // one K block = 128 bytes of a row
  int pairs = max_pairs < total_tiles ? max_pairs : total_tiles;
  // split-K tail: the tiles of a last wave that fills at most half of the pairs (all tiles, when there are so
  // few), cut into as many parts as there are pairs for, each of at least two K blocks
  p.tail_tiles = 0;
  p.tail_splits = 1;
  const int rem = total_tiles % max_pairs;
  if (a.tail_scratch != nullptr && rem > 0 && rem * 2 <= max_pairs) {
    int splits = tail_parts(rem, max_pairs, k_blocks, a.tail_splits);
    while (splits > 1 && tail_scratch_bytes(rem, splits, bn) > a.tail_scratch_bytes) --splits;
    if (splits >= 2) {
      p.tail_tiles = rem;
      p.tail_splits = splits;
      p.tail_scratch = static_cast<float*>(a.tail_scratch);
      if (total_tiles < max_pairs) pairs = rem * splits;
    }
  }
  if (a.wide_units != 0) {
    // whole waves of them (a second accumulator for each tile of a unit, so 256 columns of bf16); a pair's first work
    if (comm || fp8 || bn != 256 || a.wide_units < 0 || a.wide_units % max_pairs != 0 ||
        a.wide_units > (p.n_blocks_m + 1) / 2 * (p.n_tiles_n / 2))
      return cudaErrorInvalidValue;
    p.wide_units = a.wide_units;
  }
  const int grid = 2 * pairs;
  if (comm) {
    if (a.lead < 0) {
      // own blocks first for as long as the first round of tiles lasts: no CTA then starts the kernel
      // waiting for a peer (measured on two ranks: 693 µs with 12 own blocks first, 734 µs with 4)
      const int first_round = 2 * ((pairs + p.panel_w - 1) / p.panel_w);
      p.lead = first_round < p.blocks_per_rank ? first_round : p.blocks_per_rank;
    }
  }
  // the entry barrier of CTA i uses block slot (barrier_block_base + i): it must stay inside the block-slot region
  if (comm && ((size_t)a.barrier_block_base + grid) * a.world_size > kBlockSlots) return cudaErrorInvalidValue;
  if (p.wide_units > 0) {
    if (swiglu) return launch_wide<true, false>(ta_out, tb, tc, ta_shard, p, grid, a.overlap, stream);
    if (p.residual != nullptr) return launch_wide<false, true>(ta_out, tb, tc, ta_shard, p, grid, a.overlap, stream);
    return launch_wide<false, false>(ta_out, tb, tc, ta_shard, p, grid, a.overlap, stream);
  }
  if (swiglu && bn == 224) return launch_pair_variant<224, 7, false, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap, stream);
  if (swiglu) return launch_pair_variant<256, 6, false, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
  if (fp8) {
    switch (bn) {
      case 128: return launch_pair_variant<128, 8, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
      case 192: return launch_pair_variant<192, 7, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
      case 224: return launch_pair_variant<224, 7, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
      default:  return launch_pair_variant<256, 6, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
    }
  }
  if (p.residual != nullptr) {
    switch (bn) {
      case 128: return launch_pair_variant<128, 8, false, false, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
      case 192: return launch_pair_variant<192, 6, false, false, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
      default:  return launch_pair_variant<256, 5, false, false, true>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
    }
  }
  switch (bn) {
    case 128: return launch_pair_variant<128, 8, false>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
    case 192: return launch_pair_variant<192, 6, false>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
    case 224: return launch_pair_variant<224, 7, false>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
    default:  return launch_pair_variant<256, 6, false>(ta_shard, ta_out, tb, tc, p, grid, a.overlap && !comm, stream);
  }
}

}  // namespace smr
