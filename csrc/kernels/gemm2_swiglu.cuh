// CTA-pair tcgen05 GEMM with the SwiGLU activation in its epilogue:
//
//     act[M, F] = silu(X W_gate^T) * (X W_up^T),      W = [W_gate ; W_up] stored [2F, K]
//
// Same pipeline and barrier protocol as gemm_pair_kernel (gemm2_kernel.cuh); the
// difference is which rows of W a pair stages and what the epilogue does.  For the
// output columns [128 nb, 128 nb + 128) the leader CTA stages the gate rows
// [128 nb, +128) and its partner the up rows [F + 128 nb, +128), so the 256-column
// accumulator of every CTA holds gate in columns 0..127 and up in columns 128..255 of
// the SAME output columns: the epilogue thread that owns a row reads both, applies the
// activation on the fp32 accumulators and stores one 16-bit value.  The [M, 2F]
// intermediate is neither written nor read again (two passes over it, 4 x the size of
// the output, disappear); when the backward pass needs it (`gu` not null) it is stored
// from the same registers.  F must be a multiple of 128.  X and W are K-major.
#pragma once
#include "gemm2_kernel.cuh"

namespace ft {
namespace gemm {

template <typename T>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_pair_swiglu_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        void* act, int64_t ld_act, void* gu, int64_t ld_gu, int M,
                        int F, int K, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  PairBarriers* bars = reinterpret_cast<PairBarriers*>(smem + P_STAGES * P_STAGE_BYTES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // uniform to the compiler too
  const uint32_t cta = cluster_ctarank();            // 0 = leader
  const int pair = (int)(blockIdx.x >> 1), num_pairs = (int)(gridDim.x >> 1);
  const int mt = (M + P_BM - 1) / P_BM, nt = F / 128, kt = (K + BK - 1) / BK;
  const int num_tiles = mt * nt;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars->tmem_full[a], 1);
      mbar_init(&bars->tmem_empty[a], 8);            // 4 epilogue warps in each of the two CTAs
    }
    bars->abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile uint32_t* abort_flag = &bars->abort;
  // for the warps that work as one
  auto given_up = [&] { return __any_sync(0xffffffffu, *abort_flag != 0); };
  auto give_up = [&](int code) {
    if (lane == 0) { *abort_flag = 1; atomicCAS(err, 0, code); }
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer (both CTAs)
    int stage = 0;
    uint32_t phase = 0;
    int mb, nb;
    tile_coords(pair, mt, nt, mb, nb);
    wait_previous_kernel();
    for (int t = pair; t < num_tiles && !given_up();) {
      const int m0 = mb * P_BM + (int)cta * 128;   // this CTA's rows of X
      const int n0 = nb * 128 + (int)cta * F;      // gate rows (leader) or up rows (partner) of W
      for (int kb = 0; kb < kt; ++kb) {
        if (!mbar_wait_warp(&bars->empty[stage], phase ^ 1)) {
          give_up(21);
          break;
        }
        uint8_t* sa = smem + stage * P_STAGE_BYTES;
        uint8_t* sb = sa + P_A_BYTES;
        if (elect_one()) {
          if (cta == 0) mbar_expect_tx(&bars->full[stage], 2 * P_STAGE_BYTES);
          tma_load_2d_pair(sa, &tmap_a, &bars->full[stage], kb * BK, m0);
          tma_load_2d_pair(sb, &tmap_b, &bars->full[stage], kb * BK, n0);
        }
        __syncwarp();
        if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
      }
      t += num_pairs;
      tile_coords(t, mt, nt, mb, nb);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer (leader only)
    if (cta == 0) {
      constexpr uint32_t idesc = make_idesc_f16(std::is_same<T, __nv_bfloat16>::value ? 1 : 0, 0, 0, P_BM, P_BN);
      // descriptors of a stage are those of stage 0 plus a multiple of its size; high halves are all alike
      constexpr uint32_t A_STEP = UK * 2 >> 4, B_STEP = A_STEP;
      constexpr uint32_t dhi = smem_desc_hi(1024);
      const uint32_t a_lo = smem_desc_lo(smem_u32(smem), 16),
                     b_lo = smem_desc_lo(smem_u32(smem) + P_A_BYTES, 16);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int t = pair; t < num_tiles && !given_up(); t += num_pairs, ++it) {
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_warp(&bars->tmem_empty[acc], acc_phase ^ 1)) {
          give_up(22);
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * P_BN;
        bool failed = false;
        for (int kb = 0; kb < kt; ++kb) {
          if (!mbar_wait_warp(&bars->full[stage], phase)) {
            give_up(23);
            failed = true;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t da = a_lo + stage * (P_STAGE_BYTES >> 4), db = b_lo + stage * (P_STAGE_BYTES >> 4);
#pragma unroll
            for (int k = 0; k < BK / UK; ++k)
              umma_f16_pair(tmem_d, smem_desc_join(da + k * A_STEP, dhi), smem_desc_join(db + k * B_STEP, dhi), idesc,
                            (kb | k) != 0 ? 1u : 0u);
            umma_commit_pair(&bars->empty[stage]);
          }
          __syncwarp();
          if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
        }
        if (failed) break;
        if (elect_one()) umma_commit_pair(&bars->tmem_full[acc]);
        __syncwarp();
      }
    }
    if (lane == 0) allow_next_kernel();              // this pair's last product is under way
  } else {
    // ---------------------------------------------------------- epilogue (both CTAs)
    wait_previous_kernel();
    const int quarter = warp & 3;
    uint8_t* slots = smem + P_EPI_OFFSET + (warp - 2) * EPI_WARP_BYTES;
    // 16-byte aligned outputs whose rows are too leave by way of shared memory (see epilogue_staged); the activation alone, one
    // output of three, only over more than 512 (direct -> staged, us: 4096 x 4096 over 256 21.2 -> 23.8, 512 26.1 -> 27.2,
    // 1024 43.4 -> 42.8)
    auto aligned = [](const void* p, int64_t ld) { return ld % 8 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool staged = aligned(act, ld_act) && (gu == nullptr ? K > 512 : aligned(gu, ld_gu));
    int it = 0;
    for (int t = pair; t < num_tiles && !*abort_flag; t += num_pairs, ++it) {
      int mb, nb;
      tile_coords(t, mt, nt, mb, nb);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait_warp(&bars->tmem_full[acc], acc_phase)) {
        *abort_flag = 1;
        atomicCAS(err, 0, 24);
        break;
      }
      tc_fence_after();
      const int row = mb * P_BM + (int)cta * 128 + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + acc * P_BN + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const int col0 = nb * 128 + c * 32;          // output column (and gate column of gu)
        uint32_t g[32], u[32];
        tmem_ld_32x32(taddr + c * 32, g);
        tmem_ld_32x32(taddr + 128 + c * 32, u);
        tmem_ld_wait();
        const uint8_t* slot = slots;
        auto leave = [&](const uint32_t (&v)[32], int s) {            // one row's 32 values into slot s
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(v[8 * q + j]);
            *reinterpret_cast<uint4*>(slots + s * EPI_SLOT_BYTES + epi_unit(lane, q)) = pack8<T>(o);
          }
        };
        if (gu != nullptr) {
          if (staged) {
            leave(g, 1);
            leave(u, 2);
          } else {
            store_chunk<T, kStore16>(g, nullptr, gu, ld_gu, row, col0, M, 2 * F, ld_gu % 8 == 0, nullptr, 0, (const T*)nullptr);
            store_chunk<T, kStore16>(u, nullptr, gu, ld_gu, row, F + col0, M, 2 * F, ld_gu % 8 == 0, nullptr, 0, (const T*)nullptr);
          }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float gv = __uint_as_float(g[j]);
          g[j] = __float_as_uint(__fdividef(gv, 1.f + __expf(-gv)) * __uint_as_float(u[j]));
        }
        if (staged) {
          leave(g, 0);
          __syncwarp();
          epi_store(slot, reinterpret_cast<T*>(act), ld_act, row - lane, col0, M, F, lane);
          if (gu != nullptr) {
            epi_store(slot + EPI_SLOT_BYTES, reinterpret_cast<T*>(gu), ld_gu, row - lane, col0, M, 2 * F, lane);
            epi_store(slot + 2 * EPI_SLOT_BYTES, reinterpret_cast<T*>(gu), ld_gu, row - lane, F + col0, M, 2 * F, lane);
          }
          __syncwarp();                              // read, and free for the next columns
        } else {
          store_chunk<T, kStore16>(g, nullptr, act, ld_act, row, col0, M, F, ld_act % 8 == 0, nullptr, 0, (const T*)nullptr);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&bars->tmem_empty[acc]);
    }
  }

  tc_fence_before();
  cluster_sync_all();                                // the peer may still read this CTA's shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace gemm
}  // namespace ft
