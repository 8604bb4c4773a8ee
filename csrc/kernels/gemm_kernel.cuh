// Device side of the tcgen05 GEMM: persistent warp-specialised kernel shared by
// the plain GEMM (gemm_tcgen05.cu) and the all-gather-fused GEMM (comm/ag_gemm.cu).
// See gemm_tcgen05.cu for the description of the pipeline.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"
#include "tile_walk.cuh"
#include "../comm/peer.cuh"

namespace ft {
namespace gemm {

using namespace ft::sm100;

constexpr int BM = 128, BN = 256, BK = 64, UK = 16, STAGES = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int NUM_THREADS = 192;
constexpr int EPI_OFFSET = STAGES * STAGE_BYTES + 256;              // behind the barriers

// kAcc16Cut: as kAcc16, for rows of aligned stride whose end is no multiple of eight (columns of a wider matrix), which the way
// through shared memory cannot address; a kernel of its own, because the addends that it holds in registers ahead would
// slow the other one's epilogue down (16384 x 3072 += over 768 80 -> 98 us with four chunks of 16 columns ahead).
enum OutMode : int { kStore16 = 0, kStore32 = 1, kAcc16 = 2, kAcc32 = 3, kAcc16Cut = 4 };

// Arguments of the all-gather role of the CTA-pair kernel (gemm2_kernel.cuh, GATHER = true) and
// of the stand-alone gather (comm/ag_gemm.cu).  The gathered bytes are a window
// [w_off_bytes, w_off_bytes + w_bytes) of a flat buffer that the ranks shard in contiguous
// pieces of `shard_bytes` (rank r owns flat bytes [r * shard_bytes, (r+1) * shard_bytes));
// w_peer / w_local point at the window's first byte in every rank's / this rank's buffer.
// A row-sharded matrix is the case w_off_bytes = 0, shard_bytes = rows_per_rank * row_bytes.
// The copy warps count finished chunks per 256-row block in `ready`; the TMA producers wait for
// a block's count before they load it.
struct GatherArgs {
  peer::Peers peers;
  uint32_t seq;
  int start_slot, done_slot;
  long long spin_budget;
  const void* w_peer[peer::kMaxRanks];
  void* w_local;
  int64_t shard_bytes;     // bytes of the flat buffer each rank owns
  int64_t block_bytes;     // bytes covered by one `ready` counter
  int num_copiers;
  uint32_t* ready;
  unsigned int* block_counter;
  int64_t w_off_bytes;
  int64_t w_bytes;
  int group_m;             // CTA-pair GEMM, with or without gather: row blocks per group of the tile walk (0: GROUP_M)
  // accumulating epilogues (kAcc16 / kAcc32), with or without gather: the matrix that is added to
  // the product, of C's type and shape with row stride add_ld; nullptr = C itself (in-place +=)
  const void* add_src;
  int64_t add_ld;
  // 16-bit epilogues of two K-major operands (the forward product; the others compile without it,
  // which the weight gradients' epilogue would feel): N values of C's type added to every row, 16-byte
  // aligned; nullptr: none
  const void* bias;
  int staged;              // the epilogue goes by way of shared memory (staged_epilogue in gemm_tcgen05.cu); not with gather
  // CTA-pair GEMM with A stored MN-major and tiles of up to 128 columns, 16-bit results: the sums of A's rows
  // (over k), M values of C's type, written or, with row_sum_add, added to; nullptr: none
  void* row_sum;
  int row_sum_add;
  // CTA-pair GEMM without gather: the last split_tiles tiles of the walk are divided along the reduction
  // over split_pairs pairs (SplitWork in gemm2_kernel.cuh); split_tiles 0: none
  int split_tiles, split_pairs;
  uint64_t split_token;
  float* split_sums;       // [pairs][2 CTAs][4 warps][TN / 4 pieces][32 lanes] float4
  uint64_t* split_flags;   // [pairs][2 CTAs][4 warps]
};

// Second launch bound.  Shared memory allows one CTA per SM anyway; 3 caps the kernels at 96 registers
// a thread, which is what leaves room for two CTAs of the reduce + Adam kernel (comm/rs_adam.cu,
// 256 threads of 80) on the same SM: per scheduler 2 warps x 96 + 4 warps x 80 registers x 32
// lanes = all 16384.  The optimizer then runs under the backward pass's products.
constexpr int kMinBlocks = 3;

struct Barriers {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  uint32_t abort;
};

// Columns [col0, col0 + CW) of one output row: 16-byte stores where the chunk lies inside the matrix
// and `vec` says that the row strides keep 16-byte alignment, single elements otherwise.  `old`
// (accumulating modes, vector path) is the addend, already in registers; the element path reads it.
// `bias` (16-bit modes, or nullptr) is the row vector that is added to every row: all lanes read the
// same 16 bytes, so the pass of its own that adding it afterwards would take costs one cached load here.
template <typename T, int MODE, int CW>
__device__ __forceinline__ void store_chunk(const uint32_t (&acc)[CW], const uint4* old, void* C, int64_t ldc,
                                            int row, int col0, int M, int N, bool vec, const void* R,
                                            int64_t ldr, const T* bias) {
  if (row >= M) return;
  if constexpr (MODE == kStore32 || MODE == kAcc32) {
    float* p = reinterpret_cast<float*>(C) + (int64_t)row * ldc + col0;
    if (vec && col0 + CW <= N) {
#pragma unroll
      for (int q = 0; q < CW / 4; ++q) {
        float4 o = make_float4(__uint_as_float(acc[4 * q]), __uint_as_float(acc[4 * q + 1]),
                               __uint_as_float(acc[4 * q + 2]), __uint_as_float(acc[4 * q + 3]));
        if constexpr (MODE == kAcc32) {
          o.x += __uint_as_float(old[q].x); o.y += __uint_as_float(old[q].y);
          o.z += __uint_as_float(old[q].z); o.w += __uint_as_float(old[q].w);
        }
        reinterpret_cast<float4*>(p)[q] = o;
      }
    } else {
      const float* rp = reinterpret_cast<const float*>(R) + (int64_t)row * ldr + col0;
#pragma unroll
      for (int j = 0; j < CW; ++j)
        if (col0 + j < N) p[j] = (MODE == kAcc32 ? rp[j] : 0.f) + __uint_as_float(acc[j]);
    }
  } else {
    T* p = reinterpret_cast<T*>(C) + (int64_t)row * ldc + col0;
    if (vec && col0 + CW <= N) {
#pragma unroll
      for (int q = 0; q < CW / 8; ++q) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(acc[8 * q + j]);
        if (bias != nullptr) {
          float b[8];
          unpack8<T>(reinterpret_cast<const uint4*>(bias + col0)[q], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += b[j];
        }
        if constexpr (MODE == kAcc16 || MODE == kAcc16Cut) {
          float a[8];
          unpack8<T>(old[q], a);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += a[j];
        }
        reinterpret_cast<uint4*>(p)[q] = pack8<T>(o);
      }
    } else {
      const T* rp = reinterpret_cast<const T*>(R) + (int64_t)row * ldr + col0;
#pragma unroll
      for (int j = 0; j < CW; ++j)
        if (col0 + j < N)
          p[j] = from_float<T>((MODE == kAcc16 || MODE == kAcc16Cut ? to_float(rp[j]) : 0.f) + __uint_as_float(acc[j]) +
                               (bias != nullptr ? to_float(bias[col0 + j]) : 0.f));
    }
  }
}

// Epilogue of one warp over a 32-row x TN-column accumulator: `wait_full` blocks until the accumulator
// is complete (false: the wait ran out).
//
// The accumulating modes are bound by the latency of reading the addend, not by its bytes: with the
// loads issued 32 columns at a time behind the accumulator (and, because the addend may be C itself,
// each behind the store before it) a 256 x 256 tile spent four dependent memory latencies per 32
// columns, 33 us for a single tile, and a weight gradient over 2048 tokens (57344 x 8192 and its
// neighbours) ran at 0.58 PFLOP/s.  The addends of the first AHEAD chunks are therefore requested
// BEFORE the wait, while the tensor cores still work on the tile, and every later one AHEAD chunks
// before it is needed.  What limits AHEAD is the register budget of kMinBlocks: chunks of 16 columns
// keep the accumulator's share small, so that 96 columns (48 in fp32) of addend are in flight.  The
// modes without an addend read tensor memory one chunk ahead of the stores instead.  The same weight
// gradients now: 1.43 PFLOP/s (6.08 -> 2.43 ms), a single tile 10 us.  (Those go by way of shared memory since; what is read ahead
// here are fp32 addends and those of kAcc16Cut.  kAcc16 comes here with rows that are not aligned and with fewer than 32 columns.)
//
// BUFS: chunks of the accumulator a thread holds in the modes without an addend.  1 in the all-gather variant,
// whose seventh warp leaves fewer registers per thread (63, and two of those CTAs fit beside it as well).
template <typename T, int MODE, int TN, int BUFS, typename WaitFull>
__device__ __forceinline__ bool epilogue_tile(uint32_t taddr, void* C, int64_t ldc, int row, int tile_col0, int M,
                                              int N, const void* R, int64_t ldr, const void* bias_row,
                                              WaitFull&& wait_full) {
  const T* bias = reinterpret_cast<const T*>(bias_row);
  constexpr bool F32 = MODE == kStore32 || MODE == kAcc32;
  constexpr int ALIGN = F32 ? 4 : 8;                   // elements of 16 bytes
  if constexpr (MODE == kStore16 || MODE == kStore32) {
    const bool vec = ldc % ALIGN == 0;
    if (!wait_full()) return false;
    tc_fence_after();
    uint32_t r[BUFS][32];
    if constexpr (BUFS == 2) tmem_ld_32x32(taddr, r[0]);
#pragma unroll
    for (int c = 0; c < TN / 32; ++c) {
      const int col0 = tile_col0 + c * 32;
      if (col0 >= N) break;                            // uniform across the warp
      if constexpr (BUFS == 1) tmem_ld_32x32(taddr + c * 32, r[0]);
      tmem_ld_wait();
      if constexpr (BUFS == 2) {
        if (c + 1 < TN / 32 && col0 + 32 < N) tmem_ld_32x32(taddr + (c + 1) * 32, r[(c + 1) & 1]);
      }
      store_chunk<T, MODE>(r[c % BUFS], nullptr, C, ldc, row, col0, M, N, vec, nullptr, 0, bias);
    }
  } else {
    constexpr int CW = 16, CHUNKS = TN / CW, AHEAD = F32 ? 3 : MODE == kAcc16 ? 1 : CHUNKS < 6 ? CHUNKS : 6, W = CW / ALIGN;
    const bool vec = ldc % ALIGN == 0 && ldr % ALIGN == 0;
    const uint8_t* rp = reinterpret_cast<const uint8_t*>(R) + ((int64_t)row * ldr + tile_col0) * (F32 ? 4 : 2);
    uint4 old[AHEAD][W];
    auto request = [&](int c) {
      if (vec && row < M && tile_col0 + (c + 1) * CW <= N) {
#pragma unroll
        for (int q = 0; q < W; ++q) old[c % AHEAD][q] = reinterpret_cast<const uint4*>(rp)[c * W + q];
      }
    };
#pragma unroll
    for (int c = 0; c < AHEAD; ++c) request(c);
    if (!wait_full()) return false;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int col0 = tile_col0 + c * CW;
      if (col0 >= N) break;                            // uniform across the warp
      uint32_t r[CW];
      tmem_ld_32x16(taddr + c * CW, r);
      tmem_ld_wait();
      store_chunk<T, MODE>(r, old[c % AHEAD], C, ldc, row, col0, M, N, vec, R, ldr, bias);
      if (c + AHEAD < CHUNKS) request(c + AHEAD);
    }
  }
  return true;
}

// ---- 16-bit epilogue by way of shared memory
// A thread reads one row of the accumulator, so storing from its registers sends the 16-byte pieces of an
// instruction to 32 rows: 32 passes through the load / store unit where the 512 bytes need four, and the addend's
// loads as many again.  For a tile of 256 columns that is 4 to 8 thousand clocks of it, more than the products of a short
// reduction.  So a warp lays 32 columns of its rows out in shared memory, in a slot of 2 KB (64 bytes a row, the 16-byte
// units of eight consecutive rows on different banks), and reads and writes global memory eight whole rows at a time;
// addends arrive in the slots by cp.async, EPI_SLOTS chunks ahead and before the accumulator is complete.
// Before -> now: 50304 x 768 += over 1024 rows 85 -> 72 us, 2048 x 3072 over 768 15.9 -> 14.4.
// Three slots a warp are what leaves room for two CTAs of the reduce + Adam kernel beside a CTA of the pair kernel.
constexpr int EPI_SLOTS = 3, EPI_SLOT_BYTES = 32 * 64, EPI_WARP_BYTES = EPI_SLOTS * EPI_SLOT_BYTES;
constexpr int SMEM_BYTES = EPI_OFFSET + 4 * EPI_WARP_BYTES + 1024;
// Without the slots, for the other epilogue: what shared memory does not take is first-level cache, where a thread finds the
// rest of the 128 bytes of which it read 16 (fp32 += 4096 x 4096 over 256: 49.5 us with the slots, 48.0 without).
constexpr int SMEM_BYTES_DIRECT = EPI_OFFSET + 1024;

__device__ __forceinline__ uint32_t epi_unit(uint32_t row, uint32_t unit) {
  return row * 64 + ((unit ^ ((row >> 1) & 3)) << 4);
}

// One slot, 32 columns from `col0` of rows row0 .. row0 + 31, to global memory.
template <typename T>
__device__ __forceinline__ void epi_store(const uint8_t* slot, T* C, int64_t ldc, int row0, int col0, int M, int N,
                                          int lane) {
  const int sub = lane >> 2, unit = lane & 3, col = col0 + unit * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = sub + 8 * i;
    const uint4 v = *reinterpret_cast<const uint4*>(slot + epi_unit(r, unit));
    if (row0 + r < M && col < N) *reinterpret_cast<uint4*>(C + (int64_t)(row0 + r) * ldc + col) = v;
  }
}

// Epilogue of one warp over a 32-row x TN-column accumulator in the 16-bit modes; `slots` is the warp's own memory.
// N, ldc (and ldr) are multiples of 8 and the pointers 16-byte aligned (staged_epilogue and the launcher's checks).
template <typename T, bool ACC, int TN, typename WaitFull>
__device__ __forceinline__ bool epilogue_staged(uint32_t taddr, uint8_t* slots, T* C, int64_t ldc, int row0,
                                                int tile_col0, int M, int N, const T* R, int64_t ldr, const T* bias,
                                                int lane, WaitFull&& wait_full) {
  constexpr int CHUNKS = TN / 32;
  auto request = [&](int c) {                        // one group per chunk, empty past the end
    const int sub = lane >> 2, unit = lane & 3, col = tile_col0 + c * 32 + unit * 8;
    if (c < CHUNKS && col < N) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = sub + 8 * i;
        if (row0 + r < M)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(slots + c % EPI_SLOTS * EPI_SLOT_BYTES + epi_unit(r, unit))),
                       "l"(R + (int64_t)(row0 + r) * ldr + col)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if constexpr (ACC) {
#pragma unroll
    for (int c = 0; c < EPI_SLOTS; ++c) request(c);
  }
  const bool full = wait_full();
  if (!full) {
    if constexpr (ACC) asm volatile("cp.async.wait_all;" ::: "memory");
    return false;
  }
  tc_fence_after();
#pragma unroll 1
  for (int c = 0; c < CHUNKS; ++c) {
    const int col0 = tile_col0 + c * 32;
    if (col0 >= N) break;                            // uniform across the warp
    uint8_t* slot = slots + c % EPI_SLOTS * EPI_SLOT_BYTES;
    uint32_t r[32];
    tmem_ld_32x32(taddr + c * 32, r);
    if constexpr (ACC) {
      asm volatile("cp.async.wait_group %0;" ::"n"(EPI_SLOTS - 1) : "memory");
      __syncwarp();                                  // the other lanes' pieces too
    }
    tmem_ld_wait();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(r[8 * u + j]);
      if (bias != nullptr && col0 + u * 8 < N) {
        float b[8];
        unpack8<T>(reinterpret_cast<const uint4*>(bias + col0)[u], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += b[j];
      }
      uint4* p = reinterpret_cast<uint4*>(slot + epi_unit(lane, u));
      if constexpr (ACC) {
        float a[8];
        unpack8<T>(*p, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += a[j];
      }
      *p = pack8<T>(o);
    }
    __syncwarp();
    epi_store(slot, C, ldc, row0, col0, M, N, lane);
    if constexpr (ACC) {
      __syncwarp();                                  // every lane has read the slot
      request(c + EPI_SLOTS);
    }
  }
  if constexpr (ACC) asm volatile("cp.async.wait_all;" ::: "memory");     // of columns past the matrix: none in flight
  __syncwarp();                                      // the slots are read: the next tile may write them
  return true;
}

// ---- bulk (untiled) async copies, used by the gather role; never multicast
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void bulk_store(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                   reinterpret_cast<uint64_t>(gdst)),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all_but_1() {
  asm volatile("cp.async.bulk.wait_group 1;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void red_release_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Of `gather` this kernel uses only what its epilogue adds (it shares the launch signature of the
// CTA-pair kernel).
template <typename T, bool A_MN, bool B_MN, int MODE>
__global__ void __launch_bounds__(NUM_THREADS, kMinBlocks)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
            void* C, int64_t ldc, int M, int N, int K, int* err,
            const __grid_constant__ GatherArgs gather) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + STAGES * STAGE_BYTES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // uniform to the compiler too
  const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN, kt = (K + BK - 1) / BK;
  const int num_tiles = mt * nt;
  const int first_tile = (int)blockIdx.x;
  const int tile_step = (int)gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars->tmem_full[a], 1);
      mbar_init(&bars->tmem_empty[a], 4);
    }
    bars->abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile uint32_t* abort_flag = &bars->abort;
  // for the warps that work as one (see gemm2_kernel.cuh)
  auto given_up = [&] { return __any_sync(0xffffffffu, *abort_flag != 0); };
  auto give_up = [&](int code) {
    if (lane == 0) { *abort_flag = 1; atomicCAS(err, 0, code); }
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer
    int stage = 0;
    uint32_t phase = 0;
    int mb, nb;
    tile_coords(first_tile, mt, nt, mb, nb);
    wait_previous_kernel();
    for (int t = first_tile; t < num_tiles && !given_up();) {
      for (int kb = 0; kb < kt; ++kb) {
        if (!mbar_wait_warp(&bars->empty[stage], phase ^ 1)) {
          give_up(1);
          break;
        }
        uint8_t* sa = smem + stage * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        if (elect_one()) {
          mbar_expect_tx(&bars->full[stage], STAGE_BYTES);
          if constexpr (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_2d(sa + j * (64 * BK * 2), &tmap_a, &bars->full[stage], mb * BM + j * 64, kb * BK);
          } else {
            tma_load_2d(sa, &tmap_a, &bars->full[stage], kb * BK, mb * BM);
          }
          if constexpr (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(sb + j * (64 * BK * 2), &tmap_b, &bars->full[stage], nb * BN + j * 64, kb * BK);
          } else {
            tma_load_2d(sb, &tmap_b, &bars->full[stage], kb * BK, nb * BN);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      t += tile_step;
      tile_coords(t, mt, nt, mb, nb);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer
    constexpr uint32_t idesc =
        make_idesc_f16(sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value ? 1 : 0, A_MN ? 1 : 0,
                       B_MN ? 1 : 0, BM, BN);
    constexpr uint32_t A_STEP = (A_MN ? UK * 128 : UK * 2) >> 4, B_STEP = (B_MN ? UK * 128 : UK * 2) >> 4;
    constexpr uint32_t dhi = smem_desc_hi(1024);
    const uint32_t a_lo = smem_desc_lo(smem_u32(smem), A_MN ? 64 * BK * 2 : 16),
                   b_lo = smem_desc_lo(smem_u32(smem) + A_BYTES, B_MN ? 64 * BK * 2 : 16);
    int stage = 0;
    uint32_t phase = 0;
    int it = 0;
    for (int t = first_tile; t < num_tiles && !given_up(); t += tile_step, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait_warp(&bars->tmem_empty[acc], acc_phase ^ 1)) {
        give_up(2);
        break;
      }
      tc_fence_after();
      const uint32_t tmem_d = tmem_base + acc * BN;
      bool failed = false;
      for (int kb = 0; kb < kt; ++kb) {
        if (!mbar_wait_warp(&bars->full[stage], phase)) {
          give_up(3);
          failed = true;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t da = a_lo + stage * (STAGE_BYTES >> 4), db = b_lo + stage * (STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / UK; ++k)
            umma_f16(tmem_d, smem_desc_join(da + k * A_STEP, dhi), smem_desc_join(db + k * B_STEP, dhi), idesc,
                     (kb | k) != 0 ? 1u : 0u);
          umma_commit(&bars->empty[stage]);          // frees the stage once the MMAs have read it
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (failed) break;
      if (elect_one()) umma_commit(&bars->tmem_full[acc]);          // accumulator complete
      __syncwarp();
    }
    if (lane == 0) allow_next_kernel();              // this CTA's last product is under way
  } else {
    // ---------------------------------------------------------- epilogue
    wait_previous_kernel();
    const int quarter = warp & 3;                    // TMEM lane quarter this warp may read
    const void* add_src = gather.add_src ? gather.add_src : C;
    const int64_t add_ld = gather.add_src ? gather.add_ld : ldc;
    const bool staged = gather.staged != 0;
    int it = 0;
    for (int t = first_tile; t < num_tiles && !*abort_flag; t += tile_step, ++it) {
      int mb, nb;
      tile_coords(t, mt, nt, mb, nb);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      const int row = mb * BM + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
      auto full = [&] { return mbar_wait_warp(&bars->tmem_full[acc], acc_phase); };
      const void* bias = (A_MN || B_MN) ? nullptr : gather.bias;
      bool ok;
      if (staged) {
        if constexpr (MODE == kStore16 || MODE == kAcc16)
          ok = epilogue_staged<T, MODE == kAcc16, BN>(taddr, smem + EPI_OFFSET + (warp - 2) * EPI_WARP_BYTES,
                                                      reinterpret_cast<T*>(C), ldc, row - lane, nb * BN, M, N,
                                                      reinterpret_cast<const T*>(add_src), add_ld,
                                                      reinterpret_cast<const T*>(bias), lane, full);
      } else {
        ok = epilogue_tile<T, MODE, BN, 2>(taddr, C, ldc, row, nb * BN, M, N, add_src, add_ld, bias, full);
      }
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(err, 0, 4);
        break;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->tmem_empty[acc]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}


}  // namespace gemm
}  // namespace ft
