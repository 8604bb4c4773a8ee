// tcgen05 GEMM for products of few tiles: 16-bit results, one output tile per cluster, the reduction divided over
// one or two CTA pairs.
//
// What such a product spends its time on is not the tensor pipe: of 13 thousand clocks that a single round of
// 256 x 256 tiles over one k-block took the persistent kernel (gemm2_kernel.cuh), the next launch waited 1 700 for the
// CTAs before it to leave, 1 300 went by in the set-up, 4 800 in an epilogue of four warps and 2 000 in leaving; and 48 tiles of
// 64 columns over 3072 were bound by what an SM can load (20 KB a k-block in 337 clocks for 128 clocks of products).  So here
//   * a CTA takes half of an SM's shared memory and tensor memory at most, so that the CTAs of the next launch set
//     themselves up beside it, and two tiles of one launch run under each other's loads and epilogues;
//   * eight warps read the accumulator, and TMA moves the 16-bit tile between shared memory and the matrix: 64 columns
//     300 to 500 clocks (1 200 before);
//   * a CTA leaves without a barrier that orders memory: 100 clocks behind its last store's reads;
//   * tiles stay wide (fewer bytes a product), and a long reduction is divided over the two pairs of a cluster, each of which
//     finishes half of the columns with the other's fp32 sums (a fixed order: the same bits every time).  The sums travel through
//     distributed shared memory at some 25 bytes a clock, so that four pairs, or tiles of 256 columns, lost what they gained
//     (1024 x 768 over 3072: 8.1 us with two pairs of 128 columns, 12.5 with four of 256).
// 256 x 256 over 256: 3.8 -> 2.8 us, 2048 x 2304 over 768: 12.0 -> 7.7, 768 x 3072 += over 1024: 9.2 -> 7.4; more beside the
// rule (cluster_plan in gemm_tcgen05.cu).
//
// Cluster of 2 * splits CTAs: ranks 2 s and 2 s + 1 are pair s, which multiplies the s-th run of k-blocks.  The barriers
// full / empty / tmem_full are those of gemm2_kernel.cuh, per pair.  `addend` counts the bytes of the tile that an
// accumulating product adds, which each CTA loads for itself: without division into stages of the ring, as if they were
// k-blocks behind the last; with division behind the exchanged sums, when the ring is no longer read.  `parts` counts those sums.
// All waits are bounded; a CTA whose wait runs out records a code and takes part in the cluster barriers that are left.
#pragma once
#include "gemm2_kernel.cuh"

namespace ft {
namespace gemm {

constexpr int C_THREADS = 320;                       // producer, products, eight epilogue warps
constexpr int C_MAX_STAGES = 6;
constexpr int C_PIECE_BYTES = 128 * 64 * 2;          // 64 columns of a CTA's part of the tile, 128-byte swizzle
constexpr int C_ONES_OFFSET = 2048;                  // behind the barriers and the exchanged row sums
constexpr int C_RING_OFFSET = C_ONES_OFFSET + 2048;

struct ClusterBarriers {
  uint64_t full[C_MAX_STAGES];
  uint64_t empty[C_MAX_STAGES];
  uint64_t tmem_full, addend, parts;
  uint32_t tmem_base;
  uint32_t late;           // an epilogue warp's wait ran out
};
constexpr int C_SUMS_OFFSET = 256;                   // 128 row sums of the other pair
static_assert(sizeof(ClusterBarriers) <= C_SUMS_OFFSET && C_SUMS_OFFSET + 512 <= C_ONES_OFFSET, "layout");

// Bytes of a stage: a CTA's 128 rows of A and its half of B (whole chunks of 64 columns where B is MN-major).
__host__ __device__ constexpr int cluster_stage_bytes(int tn, bool b_mn) {
  return P_A_BYTES + (b_mn ? (tn / 2 + 63) / 64 * 64 : tn / 2) * BK * 2;
}

// Columns of tensor memory: the tile's and, in tiles of up to 192 columns, 32 for the row sums, a power of TWO.
constexpr int C_SUMS_TILE = 192;
__host__ __device__ constexpr int cluster_tmem_columns(int tn, bool sums) {
  const int n = tn + (sums ? 32 : 0);
  return n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}

struct ClusterArgs {
  int M, N, K;
  int splits;              // pairs of a cluster: 1, or 2 with tiles of 128 columns
  int stages, first_stage; // of the ring, and the one behind the last k-block's where the reduction is not divided
  int mt, nt, kt, group_m;
  const void* bias;        // K-major operands: N values added to every row; nullptr: none
  void* row_sum;           // both operands MN-major: sums of A's rows over k (see GatherArgs); nullptr: none
  int row_sum_add;
  int* err;
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// 16 bytes to another CTA of the cluster, counted by its barrier
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(x),
               "r"(y), "r"(z), "r"(w), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem)), "r"(x), "r"(y)
               : "memory");
}

__device__ __forceinline__ uint4 ld_shared(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void st_shared(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// The 256 threads of the epilogue warps
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// Commit whose arrival both CTAs of a pair receive, whose leader has `rank`.
__device__ __forceinline__ void umma_commit_ranks(uint64_t* bar, uint32_t rank) {
  const uint16_t mask = (uint16_t)(3u << rank);
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(mask)
      : "memory");
}

// One CTA's part of a product, whose clusters are numbered from `block` = 0 on.
// ACC: `tmap_r` is the matrix that is added, of C's shape (C itself for +=).  Both maps have boxes of 64 columns x 128 rows.
template <typename T, bool A_MN, bool B_MN, bool ACC, int TN>
__device__ __forceinline__ void cluster_product(const CUtensorMap& tmap_a, const CUtensorMap& tmap_b, const CUtensorMap& tmap_c,
                                                const CUtensorMap& tmap_r, const ClusterArgs& args, int block) {
  constexpr int STAGE = cluster_stage_bytes(TN, B_MN), TWO = TN == 256 ? 1 : 0;      // a stage holds 1 + TWO pieces
  constexpr bool SUMS = A_MN && B_MN && TN <= C_SUMS_TILE, SPLIT = TN == 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  ClusterBarriers* bars = reinterpret_cast<ClusterBarriers*>(smem);
  uint8_t* ring = smem + C_RING_OFFSET;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), cta = rank & 1;
  const int splits = SPLIT ? args.splits : 1, split = SPLIT ? (int)rank >> 1 : 0;
  const int M = args.M, N = args.N, stages = args.stages, kt = args.kt;
  const int kb0 = splits == 1 ? 0 : kt * split >> 1, kb1 = splits == 1 ? kt : kt * (split + 1) >> 1;
  int mb, nb;
  tile_coords(block >> splits, args.mt, args.nt, mb, nb, args.group_m);
  const int m0 = mb * P_BM + (int)cta * 128;         // this CTA's rows
  const bool row_sums = SUMS && args.row_sum != nullptr && nb == 0;
  // pieces of the tile that this CTA finishes: all, or its share of a divided tile, those inside the matrix
  const int own = TN >> (5 + splits), col0 = nb * TN + split * own * 64;
  const int pieces = min(own, (N - col0 + 63) / 64);

  const uint32_t tmem_cols = cluster_tmem_columns(TN, row_sums);      // alike in both CTAs of a pair

  if constexpr (SUMS) {
    if (row_sums && threadIdx.x < P_ONES_BYTES / 16) {
      const float one[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
      reinterpret_cast<uint4*>(smem + C_ONES_OFFSET)[threadIdx.x] = pack8<T>(one);
      fence_proxy_async();
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->tmem_full, 1);
    mbar_init(&bars->addend, 1);
    mbar_init(&bars->parts, 1);
    bars->late = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    prefetch_tmap(&tmap_c);
    if constexpr (ACC) prefetch_tmap(&tmap_r);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, tmem_cols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  auto give_up = [&](int code) {
    if (lane == 0) atomicCAS(args.err, 0, code);
  };
  // Where the pieces of what this CTA finishes lie in shared memory.  Undivided: in the stages behind the last k-block's, in the
  // order in which the products leave them.  Divided: behind the sums of the other pairs.
  const int exchange = (splits - 1) * own * (128 * 64 * 4), first_stage = args.first_stage;
  auto piece = [&](int p) -> uint8_t* {
    if (splits > 1) return ring + exchange + p * C_PIECE_BYTES;
    int stage = first_stage + (p >> TWO);
    if (stage >= stages) stage -= stages;
    return ring + stage * STAGE + (p & TWO) * C_PIECE_BYTES;
  };

  const int quarter = warp & 3, half = (warp - 2) >> 2;         // of an epilogue warp: its rows, and which half of each piece
  const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
  bool complete = false;                             // epilogue warps: the accumulator is

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer (every CTA)
    wait_previous_kernel();
    const int n0 = nb * TN + (int)cta * (TN >> 1);        // this CTA's half of B
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&bars->empty[stage], phase ^ 1)) { give_up(31); ok = false; break; }
      uint8_t* sa = ring + stage * STAGE;
      uint8_t* sb = sa + P_A_BYTES;
      if (elect_one()) {
        if (cta == 0) mbar_expect_tx(&bars->full[stage], 2 * STAGE);
        if constexpr (A_MN) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
            tma_load_2d_pair(sa + j * (64 * BK * 2), &tmap_a, &bars->full[stage], m0 + j * 64, kb * BK);
        } else {
          tma_load_2d_pair(sa, &tmap_a, &bars->full[stage], kb * BK, m0);
        }
        if constexpr (B_MN) {
#pragma unroll
          for (int j = 0; j < (TN > 128 ? 2 : 1); ++j)
            tma_load_2d_pair(sb + j * (64 * BK * 2), &tmap_b, &bars->full[stage], n0 + j * 64, kb * BK);
        } else {
          tma_load_2d_pair(sb, &tmap_b, &bars->full[stage], kb * BK, n0);
        }
      }
      __syncwarp();
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
    if constexpr (ACC) {
      // the addend follows the operands through the ring: on its way while the last products run
      if (splits == 1 && ok) {
        if (elect_one()) mbar_expect_tx(&bars->addend, pieces * C_PIECE_BYTES);
        __syncwarp();
        for (int p = 0; p < pieces; p += 1 + TWO) {
          if (!mbar_wait_warp(&bars->empty[stage], phase ^ 1)) { give_up(31); break; }
          if (elect_one()) {
            for (int q = p; q <= p + TWO && q < pieces; ++q)
              tma_load_2d(piece(q), &tmap_r, &bars->addend, col0 + q * 64, m0);
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- products (a pair's leader)
    if (cta == 0) {
      constexpr int format = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      constexpr uint32_t idesc = make_idesc_f16(format, A_MN ? 1 : 0, B_MN ? 1 : 0, P_BM, TN);
      constexpr uint32_t idesc_sum = make_idesc_f16(format, A_MN ? 1 : 0, 0, P_BM, 32);
      constexpr uint32_t A_STEP = (A_MN ? UK * 128 : UK * 2) >> 4, B_STEP = (B_MN ? UK * 128 : UK * 2) >> 4;
      constexpr uint32_t dhi = smem_desc_hi(1024);
      const uint32_t a_lo = smem_desc_lo(smem_u32(ring), A_MN ? 64 * BK * 2 : 16),
                     b_lo = smem_desc_lo(smem_u32(ring) + P_A_BYTES, B_MN ? 64 * BK * 2 : 16),
                     ones = smem_desc_lo(smem_u32(smem) + C_ONES_OFFSET, 16);
      const int behind = ACC && splits == 1 ? (pieces + TWO) >> TWO : 0;      // stages of the addend
      const int last_waited = kb1 + behind - stages;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&bars->full[stage], phase)) { give_up(32); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t da = a_lo + stage * (STAGE >> 4), db = b_lo + stage * (STAGE >> 4);
#pragma unroll
          for (int k = 0; k < BK / UK; ++k)
            umma_f16_pair(tmem_base, smem_desc_join(da + k * A_STEP, dhi), smem_desc_join(db + k * B_STEP, dhi), idesc,
                          kb != kb0 || k != 0 ? 1u : 0u);
          if constexpr (SUMS) {
            if (row_sums) {
#pragma unroll
              for (int k = 0; k < BK / UK; ++k)
                umma_f16_pair(tmem_base + TN, smem_desc_join(da + k * A_STEP, dhi), smem_desc_join(ones, dhi), idesc_sum,
                              kb != kb0 || k != 0 ? 1u : 0u);
            }
          }
          // only where a producer waits for it: no arrival is under way to a CTA that may have left
          if (kb < last_waited) umma_commit_ranks(&bars->empty[stage], rank);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
      if (ok && elect_one()) umma_commit_ranks(&bars->tmem_full, rank);
      __syncwarp();
    }
    if (lane == 0) allow_next_kernel();
  } else {
    wait_previous_kernel();
    if (!mbar_wait_warp(&bars->tmem_full, 0)) {
      give_up(33);
      if (lane == 0) bars->late = 1;
    }
    epilogue_sync();                                 // one verdict for the eight warps
    complete = *reinterpret_cast<volatile uint32_t*>(&bars->late) == 0;
    tc_fence_after();
  }

  if (splits > 1) {
    cluster_sync_all();                            // nobody's ring is read any more
    if (warp >= 2 && complete) {
      if constexpr (ACC) {
        if (threadIdx.x == 64) {
          fence_proxy_async();
          mbar_expect_tx(&bars->addend, max(pieces, 0) * C_PIECE_BYTES);
          for (int p = 0; p < pieces; ++p) tma_load_2d(piece(p), &tmap_r, &bars->addend, col0 + p * 64, m0);
        }
        __syncwarp();
      }
      // the other pair's columns to its CTA of the same rows, [column / 4][row] float4: 16 columns at a time
      const uint32_t to = rank ^ 2, bar = map_to_rank(smem_u32(&bars->parts), to),
                     base = map_to_rank(smem_u32(ring), to) + (half * 8 * 128 + quarter * 32 + lane) * 16;
      const uint32_t from = taddr + (split ^ 1) * own * 64 + half * 32;
      if (threadIdx.x == 64) mbar_expect_tx(&bars->parts, own * 64 * 128 * 4);
      uint32_t r[32];
#pragma unroll 1
      for (int p = 0; p < own; ++p) {
        tmem_ld_32x32(from + p * 64, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          st_async(base + (16 * p + q) * 2048, r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3], bar);
      }
      if constexpr (SUMS) {
        if (row_sums && split > 0 && half == 0) {
          uint32_t s[16];
          tmem_ld_32x16(taddr + TN, s);
          tmem_ld_wait();
          const uint32_t sum = map_to_rank(smem_u32(smem + C_SUMS_OFFSET), cta) + (quarter * 32 + lane) * 4;
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(sum), "r"(s[0]) : "memory");
        }
      }
    }
    if constexpr (SUMS) {
      if (row_sums) cluster_sync_all();
    }
  }

  if (warp >= 2 && complete) {
    // ---------------------------------------------------------- epilogue
    const int row = quarter * 32 + lane;
    const T* bias = (A_MN || B_MN) ? nullptr : reinterpret_cast<const T*>(args.bias);
    bool ok = true;
    if (splits > 1 && !mbar_wait_warp(&bars->parts, 0)) { ok = false; give_up(35); }
    if constexpr (ACC) {
      if (pieces > 0) ok &= mbar_wait_warp(&bars->addend, 0);
      if (!ok) give_up(34);
    }
    const uint32_t mine = taddr + split * own * 64 + half * 32;
    // 16 columns of this thread's row, the h-th of this warp's in piece p
    auto finish = [&](uint32_t (&r)[16], int p, int h) {
      if (splits > 1) {                              // the sums of the other pair
        const uint32_t part = smem_u32(ring) + ((16 * p + half * 8 + h * 4) * 128 + row) * 16;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 v = ld_shared(part + q * 2048);
          r[4 * q] = __float_as_uint(__uint_as_float(r[4 * q]) + __uint_as_float(v.x));
          r[4 * q + 1] = __float_as_uint(__uint_as_float(r[4 * q + 1]) + __uint_as_float(v.y));
          r[4 * q + 2] = __float_as_uint(__uint_as_float(r[4 * q + 2]) + __uint_as_float(v.z));
          r[4 * q + 3] = __float_as_uint(__uint_as_float(r[4 * q + 3]) + __uint_as_float(v.w));
        }
      }
      const int col = col0 + p * 64 + half * 32 + h * 16;
      const uint32_t at = smem_u32(piece(p)) + row * 128;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t unit = at + (((half * 4 + h * 2 + u) ^ (row & 7)) << 4);
        float o[8], a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(r[8 * u + j]);
        if (bias != nullptr && col + u * 8 < N) {
          unpack8<T>(*reinterpret_cast<const uint4*>(bias + col + u * 8), a);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += a[j];
        }
        if constexpr (ACC) {
          unpack8<T>(ld_shared(unit), a);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += a[j];
        }
        st_shared(unit, pack8<T>(o));
      }
    };
    // the next 16 columns leave tensor memory while these are converted
    uint32_t ra[16], rb[16];
    if (pieces > 0) tmem_ld_32x16(mine, ra);
#pragma unroll 1
    for (int p = 0; p < pieces; ++p) {
      tmem_ld_wait();
      tmem_ld_32x16(mine + p * 64 + 16, rb);
      finish(ra, p, 0);
      tmem_ld_wait();
      if (p + 1 < pieces) tmem_ld_32x16(mine + p * 64 + 64, ra);
      finish(rb, p, 1);
      fence_proxy_async();
      epilogue_sync();
      if (ok && threadIdx.x == 64 && m0 < M) {
        tma_store_2d(&tmap_c, piece(p), col0 + p * 64, m0);
        bulk_commit();
      }
    }
    if constexpr (SUMS) {
      if (row_sums && split == 0 && half == 0) {
        uint32_t s[16];                              // alike: one column per one
        tmem_ld_32x16(taddr + TN, s);
        tmem_ld_wait();
        float sum = __uint_as_float(s[0]);
        if (splits > 1) sum += reinterpret_cast<const float*>(smem + C_SUMS_OFFSET)[row];
        if (m0 + row < M) {
          T* out = reinterpret_cast<T*>(args.row_sum) + m0 + row;
          *out = from_float<T>(sum + (args.row_sum_add ? to_float(*out) : 0.f));
        }
      }
    }
  }

  // Nobody reads or writes this CTA's memory from elsewhere any more (products and exchanged sums have been waited for); what
  // the pair waits for here is the release of its tensor memory.  The arrival is early and orders nothing else: as
  // a barrier behind the store's wait, with release, it took 1 100 to 1 300 clocks.
  tc_fence_before();
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  if (threadIdx.x == 64) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
  asm volatile("barrier.cluster.wait;" ::: "memory");
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, tmem_cols);
  }
}

template <typename T, bool A_MN, bool B_MN, bool ACC, int TN>
__global__ void __launch_bounds__(C_THREADS, 2)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_r,
                    const __grid_constant__ ClusterArgs args) {
  cluster_product<T, A_MN, B_MN, ACC, TN>(tmap_a, tmap_b, tmap_c, tmap_r, args, (int)blockIdx.x);
}

// The two products of a projection's backward pass in one launch, dX = dY W and dW (+)= dY^T X (with dY's column sums): neither fills the
// machine in whole rounds, and each would start and drain by itself.  The first `first_blocks` CTAs take dW where `dw_first`, the
// longer reduction, and dX otherwise.
template <typename T, bool ACC, int TN>
__global__ void __launch_bounds__(C_THREADS, 2)
gemm_cluster_backward_kernel(const __grid_constant__ CUtensorMap dy_rows, const __grid_constant__ CUtensorMap w,
                             const __grid_constant__ CUtensorMap dx, const __grid_constant__ CUtensorMap dy_columns,
                             const __grid_constant__ CUtensorMap x, const __grid_constant__ CUtensorMap dw,
                             const __grid_constant__ ClusterArgs dx_args, const __grid_constant__ ClusterArgs dw_args,
                             int first_blocks, int dw_first) {
  const bool first = (int)blockIdx.x < first_blocks;
  const int block = (int)blockIdx.x - (first ? 0 : first_blocks);
  if (first == (dw_first != 0)) cluster_product<T, true, true, ACC, TN>(dy_columns, x, dw, dw, dw_args, block);
  else cluster_product<T, false, true, false, TN>(dy_rows, w, dx, dx, dx_args, block);
}

}  // namespace gemm
}  // namespace ft
