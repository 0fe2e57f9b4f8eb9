// GEMM on pairs of CTAs (cta_group::2): 256 x BN output tiles.
//
// What bounds the one-CTA kernel (gemm_kernel.cuh) is shared memory: per k-block of 64 a 128 x 256 tile writes 48 KiB by TMA and reads them
// once for 512 cycles of tensor work, 768 cycles at 128 bytes a clock. A pair shares the B operand: each CTA stages its own 128 rows of
// A and half of B's columns, so 32 KiB in and 32 KiB out serve the same 512 cycles.
//
// Both CTAs run a TMA warp; all loads of a stage complete on the leader's `full` barrier, which the leader alone arms. The leader's MMA warp
// issues for both and frees a stage, and hands over an accumulator, by a commit that arrives at both CTAs' barriers. Each CTA's
// epilogue stores its own 128 rows; its eight warps (two per TMEM lane quadrant, half of the columns each) arrive at the leader's `tempty`.
#pragma once
#include "gemm_kernel.cuh"

namespace ra {
namespace gemm {

constexpr int PAIR_EPI_WARPS = 8;
constexpr int PAIR_THREADS = 64 + 32 * PAIR_EPI_WARPS;

template <int BN_>
struct PairTile {
  static constexpr int STAGES = BN_ == 256 ? 6 : 8;
  static constexpr int A_STAGE_BYTES = BM * BK * 2;          // this CTA's rows
  static constexpr int B_STAGE_BYTES = BN_ / 2 * BK * 2;     // this CTA's half of the columns
  static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + PAIR_EPI_WARPS * EPI_STAGE + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr int TMEM_COLS = NUM_ACC * BN_;
};

template <int A_MN, int B_MN, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const Params p) {
  using T = PairTile<BN>;
  constexpr int STAGES = T::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * T::A_STAGE_BYTES;
  uint8_t* sE = sB + STAGES * T::B_STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(sE + PAIR_EPI_WARPS * EPI_STAGE);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + NUM_ACC;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + NUM_ACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const WaitCtx wc{abort_flag, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < NUM_ACC; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 2 * PAIR_EPI_WARPS);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, T::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the other CTA's barriers are there too
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int tiles_n = p.swiglu_F ? (p.swiglu_F + BN / 2 - 1) / (BN / 2) : (p.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = (p.K + BK - 1) / BK;
  const int group_m = p.group_m > 1 ? p.group_m / 2 : 1;
  const int first = static_cast<int>(blockIdx.x) >> 1, step = static_cast<int>(gridDim.x) >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs, warp-uniform flow)
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    // Behind the last tile it waits for every stage once more (one that was never filled passes at once): the leader's commits arrive at both
    // CTAs' `empty`, and nothing orders one commit's arrivals before a later one's, so the last of them could otherwise reach a CTA that has
    // seen its last accumulator and left.
    bool more = true;
    for (int tile = first; more && ok; tile += step) {
      more = tile < num_tiles;
      const int steps = more ? num_kb : STAGES;
      int tm, tn;
      tile_coords(tile, tiles_m, tiles_n, group_m, tm, tn);
      const int m0 = (2 * tm + static_cast<int>(rank)) * BM;
      // with SwiGLU the leader's columns are the gate's and the other CTA's the matching ones of up
      const int n0 = p.swiglu_F ? static_cast<int>(rank) * p.swiglu_F + tn * (BN / 2) : tn * BN + static_cast<int>(rank) * (BN / 2);
      for (int kb = 0; kb < steps; ++kb) {
        const int k0 = kb * BK;
        if (!mbar_wait(&empty[stage], phase ^ 1u, wc, kTimeoutSmemEmpty)) {
          ok = false;
          break;
        }
        uint8_t* a_dst = sA + stage * T::A_STAGE_BYTES;
        uint8_t* b_dst = sB + stage * T::B_STAGE_BYTES;
        const uint32_t bar = cluster_map(&full[stage], 0);
        if (elected && more) {
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * T::STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i) tma_load_2d_pair(a_dst + i * SLAB_BYTES, &tma_a, bar, m0 + 64 * i, k0);
          } else {
            tma_load_2d_pair(a_dst, &tma_a, bar, k0, m0);
          }
          if (B_MN) {
#pragma unroll
            for (int i = 0; i < BN / 128; ++i) tma_load_2d_pair(b_dst + i * SLAB_BYTES, &tma_b, bar, n0 + 64 * i, k0);
          } else {
            tma_load_2d_pair(b_dst, &tma_b, bar, k0, n0);
          }
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the leader's, warp-uniform flow)
    if (rank == 0) {
      const bool elected = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        if (!mbar_wait_cluster(&tempty[acc], acc_phase ^ 1u, wc, kTimeoutTmemEmpty)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase, wc, kTimeoutSmemFull)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(sA + stage * T::A_STAGE_BYTES);
          const uint32_t b_addr = smem_u32(sB + stage * T::B_STAGE_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const uint64_t adesc = A_MN ? make_smem_desc(a_addr + kk * 2048, SLAB_BYTES, 1024)
                                        : make_smem_desc(a_addr + kk * 32, 16, 1024);
            const uint64_t bdesc = B_MN ? make_smem_desc(b_addr + kk * 2048, SLAB_BYTES, 1024)
                                        : make_smem_desc(b_addr + kk * 32, 16, 1024);
            if (elected) umma_ss_pair(d_tmem, adesc, bdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          if (elected) umma_commit_pair(&empty[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (elected) umma_commit_pair(&tfull[acc]);
        if (++acc == NUM_ACC) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;           // TMEM lane quadrant this warp may access
    const int half = (warp - 2) >> 2;    // of the columns
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = first; tile < num_tiles; tile += step) {
      int tm, tn;
      tile_coords(tile, tiles_m, tiles_n, group_m, tm, tn);
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * BN);
      // a wait that gives up ends the loop for the whole warp: the TMEM loads behind it are warp-collective
      if (!epilogue<BN>(p, t_row, (2 * tm + static_cast<int>(rank)) * BM + quad * 32, tn, half * (BN / 64), (half + 1) * (BN / 64),
                        sE + (warp - 2) * EPI_STAGE,
                        [&] { return __all_sync(0xffffffffu, mbar_wait(&tfull[acc], acc_phase, wc, kTimeoutTmemFull)); }))
        break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_map(&tempty[acc], 0));
      if (++acc == NUM_ACC) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) bounded_drain_pause();
  cluster_arrive();  // neither CTA's shared memory or TMEM goes while the other still uses it
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, T::TMEM_COLS);
  }
}

}  // namespace gemm
}  // namespace ra
