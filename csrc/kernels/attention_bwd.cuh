// Causal grouped-query flash attention, backward, on tcgen05 tensor cores.
//
// One CTA per (batch, kv head, 128-row kv block n).  K_n and V_n stay in shared
// memory; the CTA walks every query head of the group and every query block
// m >= n, and per (head, m), a step:
//   TMA      Q_m, dO_m                      ([64-col chunk][row][64], 128B swizzle)
//   MMA      S^T = K Q^T,  dP^T = V dO^T    -> TMEM, a kv row per lane
//   warps    P^T = exp(scale*S^T - lse), written over S^T as packed 16-bit pairs;
//            dS^T = P^T * (dP^T - delta), as a 16-bit tile [kv][q] into shared memory.  lse and
//            delta belong to columns here and are read from a small shared-memory table.  The
//            softmax scale is not applied to dS: dK is scaled once when it is written and dQ by
//            the conversion pass.
//   MMA      dV += P^T dO (P^T straight from tensor memory), dK += dS^T Q (both accumulated in
//            TMEM over the whole walk), dQ_m = dS K -> over dP^T in TMEM -> fp32 slabs in shared
//            memory (half of them in memory of their own, half in the dS tile, idle by then) -> one
//            TMA reduce-add per 32-column slab into dq_acc, issued by a dedicated warp
// Consecutive steps overlap: S^T of the next step is computed as soon as dV has consumed P^T, so the
// next exponentials run under dK and dQ, and dP^T of the next step follows as soon as dQ has left its
// columns.  The order of the tensor pipe is
//            dP(i) dV(i) S(i+1) dK(i) dQ(i) dP(i+1) ...
// With S, softmax, dV, dP, dS, dK, dQ and its read-out one after the other (and P as a second shared-memory
// tile) a step of 128 x 128 x 128 took 5 990 clocks, 2 560 of them products; now 5 500.  Heads of 64: 50 -> 41 us for
// 3 x 1000 tokens of 16.  What bounds it at head size 128 are the reduce-adds: the 64 KB of a dQ tile keep the TMA unit
// busy for 3 260 clocks, dS waits for the slabs in its tile to be read (1 400) and dO's load queues behind them.  Adding
// from registers instead (red.v4, lane pairs on one sector, no slabs) took 5 500 clocks a tile, 9 050 a step.
// dO is released for the next load as soon as dV is complete; Q has two buffers, because S(i+1) is
// computed before dK(i).
// The same shared-memory bytes serve as K-major operand (reduction over the 64
// contiguous columns) and as MN-major operand (reduction over the rows), so no
// tile is ever transposed.  dK / dV are written once at the end; dq_acc is
// converted to the 16-bit dq by a separate pass.  All waits are bounded.
#pragma once
#include "attention_common.cuh"
#include "packed_math.cuh"

namespace ft {
namespace attn {

// 2 control warps + 4 * SPLIT compute warps + the dQ store warp.  The 128 columns of S / dP (and
// the D columns of dQ / dK / dV) are cut into SPLIT parts; warps 2 + 4 * part .. 5 + 4 * part own
// part `part` (each warp still reads only its own TMEM lane quarter, warp % 4), so every score
// row is shared by SPLIT threads.  The warp after them issues the dQ reduce-adds.
constexpr int bwd_threads(int split) { return 32 * (2 + 4 * split + 1); }

template <int D>
struct BwdSmem {
  static constexpr int TILE = BQ * D * 2;
  static constexpr int DS_BYTES = BQ * BKV * 2;
  // dQ leaves through fp32 slabs of [128 rows][32 columns] (16 KB each).  At head size 128 the
  // first two have shared memory of their own and the last two reuse the dS tile, which is idle
  // between the dQ product and the next dS; at head size 64 both slabs have their own.
  static constexpr int SLAB = BQ * 128;
  static constexpr int OWN_SLABS = 2;
  static constexpr int STAT_BYTES = 2 * 2 * BQ * 4;  // two stages of -lse * log2(e) and -delta
  // K, V, two of Q, dO; nothing is left for an alignment gap at head size 128 (the base is checked)
  static constexpr int BYTES = 5 * TILE + DS_BYTES + OWN_SLABS * SLAB + STAT_BYTES + 256;
};

struct BwdBars {
  uint64_t kv_full, q_full[2], q_empty[2], do_full, do_empty, stat_full[2];
  uint64_t s_full, dp_full, p_full, ds_full, dq_full, dq_read, acc_full;
  uint64_t dqs_full, own_free, shared_free;
  uint32_t tmem_base;
  uint32_t abort;
};
static_assert(sizeof(BwdBars) <= 256, "barrier block outgrew its slot");

struct BwdParams {
  const float* lse;        // [B, Hq, S]
  const float* delta;      // [B, Hq, S]  rowsum(dO * O)
  float* dq_acc;           // [B, S, Hq, D] fp32, zeroed by the caller
  void* dk; int64_t dk_stride;   // [B, S, Hkv, D] with token stride
  void* dv; int64_t dv_stride;
  int B, S, Hq, Hkv;
  int chunk;               // (batch, kv head, part) groups per chunk of the CTA order (causal_job)
  // The query heads of a kv head are divided over `splits` CTAs of `part_heads` heads each (the last
  // may have fewer).  One part: dk and dv are written directly.  More: each part leaves its fp32 sums in
  // kv_part [splits][2: dk, dv][B * S][Hkv * D], which attn_dkv_sum_kernel adds up.
  int splits, part_heads;
  float* kv_part;
  float scale, scale_log2;
  int* err;
  // timeline capture (TRACE instantiation only): clock64() of CTA trace_cta at the hand-over points
  // of iterations trace_it0 .. trace_it0 + 7, as trace[(role * 16 + site) * 8 + iteration]
  long long* trace;
  int trace_cta, trace_it0;
};

// fp32 tile in shared memory (128B-swizzled [rows][32] slab) added into global memory
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* smem_src, int32_t x,
                                                  int32_t y) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(m)),
      "r"(smem_u32(smem_src)), "r"(x), "r"(y)
      : "memory");
}

// POLY: which of every eight pairs of P values take the polynomial 2^x (bit j = pair j); the
// rest use the special-function unit, so both pipes work on one score row.
template <typename T, int D, int SPLIT, bool TRACE = false, unsigned POLY = 0xAAu>
__global__ void __launch_bounds__(bwd_threads(SPLIT), 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const __grid_constant__ CUtensorMap tmap_dq, const __grid_constant__ BwdParams P) {
  constexpr int TILE = BwdSmem<D>::TILE;
  constexpr int CHUNKS = D / 64;
  constexpr int CHUNK_BYTES = BQ * 128;
  extern __shared__ __align__(1024) uint8_t bwd_smem[];
  uint8_t* sK = bwd_smem;
  uint8_t* sV = sK + TILE;
  uint8_t* sQ = sV + TILE;                           // two stages
  uint8_t* sdO = sQ + 2 * TILE;
  uint8_t* sdS = sdO + TILE;
  uint8_t* sStage = sdS + BwdSmem<D>::DS_BYTES;
  float* sStat = reinterpret_cast<float*>(sStage + BwdSmem<D>::OWN_SLABS * BwdSmem<D>::SLAB);
  BwdBars* bars = reinterpret_cast<BwdBars*>(sStat + 4 * BQ);
  constexpr int OWN_SLABS = BwdSmem<D>::OWN_SLABS;
  if (smem_u32(bwd_smem) & 1023) {                   // the swizzle goes by address bits
    if (threadIdx.x == 0) atomicCAS(P.err, 0, 416);
    return;
  }
  // fp32 slab c of the dQ tile
  auto slab_ptr = [&](int c) -> uint8_t* {
    return c < OWN_SLABS ? sStage + c * BwdSmem<D>::SLAB : sdS + (c - OWN_SLABS) * BwdSmem<D>::SLAB;
  };

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_blk = (P.S + BQ - 1) / BQ;
  const CausalJob job = causal_job((int)blockIdx.x, P.B * P.Hkv * P.splits, num_blk, P.chunk);
  const int nb = job.rank;                           // kv block; low blocks (most work) first
  const int kv_head = (job.head / P.splits) % P.Hkv;
  const int batch = job.head / (P.splits * P.Hkv);
  const int group = P.Hq / P.Hkv;
  const int head0 = kv_head * group + (job.head % P.splits) * P.part_heads;    // first query head of this CTA
  const int q_blocks = num_blk - nb;                 // m = nb .. num_blk-1
  const int iters = min(P.part_heads, (kv_head + 1) * group - head0) * q_blocks;
  const int kv_row0 = batch * P.S + nb * BKV;
  // role: 0 loads, 1 products, 2 first softmax warp, 3 last softmax warp, 4 dQ reduce warp
  auto stamp = [&](int role, int site, int it) {
    if constexpr (TRACE) {
      if ((int)blockIdx.x == P.trace_cta && it >= P.trace_it0 && it < P.trace_it0 + 8)
        P.trace[(role * 16 + site) * 8 + (it - P.trace_it0)] = clock64();
    }
  };

  if (threadIdx.x == 0) {
    mbar_init(&bars->kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->q_full[s], 1);
      mbar_init(&bars->q_empty[s], 1);
      mbar_init(&bars->stat_full[s], 32);
    }
    mbar_init(&bars->do_full, 1);
    mbar_init(&bars->do_empty, 1);
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->p_full, 128 * SPLIT);
    mbar_init(&bars->ds_full, 128 * SPLIT);
    mbar_init(&bars->dq_full, 1);
    mbar_init(&bars->dq_read, 128 * SPLIT);
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->dqs_full, 128 * SPLIT);
    mbar_init(&bars->own_free, 1);
    mbar_init(&bars->shared_free, 1);
    bars->abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v); prefetch_tmap(&tmap_do);
    prefetch_tmap(&tmap_dq);
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile uint32_t* abort_flag = &bars->abort;
  wait_previous_kernel();
  const uint32_t tm_s = tmem, tm_dp = tmem + 128, tm_dv = tmem + 256, tm_dk = tmem + 384;
  const uint32_t tm_dq = tm_dp;                      // reuses the dP columns once dS is written

  const float log2e = 1.4426950408889634f;
  if (warp == 0) {
    // ------------------------------------------------------------ loads (the whole warp)
    auto row_of = [&](int it, int& head) {           // first query row of step `it`, in its sequence
      head = head0 + it / q_blocks;
      return (nb + it % q_blocks) * BQ;
    };
    auto load_q = [&](int it) {
      int head;
      const int row = row_of(it, head), s = it & 1;
      if (elect_one()) {
        mbar_expect_tx(&bars->q_full[s], TILE);
        for (int c = 0; c < CHUNKS; ++c)
          tma_load_2d(sQ + s * TILE + c * CHUNK_BYTES, &tmap_q, &bars->q_full[s], head * D + c * 64, batch * P.S + row);
      }
      __syncwarp();
    };
    auto load_do = [&](int it) {
      int head;
      const int row = row_of(it, head);
      if (elect_one()) {
        mbar_expect_tx(&bars->do_full, TILE);
        for (int c = 0; c < CHUNKS; ++c)
          tma_load_2d(sdO + c * CHUNK_BYTES, &tmap_do, &bars->do_full, head * D + c * 64, batch * P.S + row);
      }
      __syncwarp();
    };
    // columns past the end of the sequence: lse = +inf makes every P (and dS) of the column zero
    auto load_stats = [&](int it) {
      int head;
      const int row = row_of(it, head);
      const int64_t first = ((int64_t)batch * P.Hq + head) * P.S + row;
      float* out = sStat + (it & 1) * 2 * BQ;
      float l[4], d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = j * 32 + lane;
        const bool ok = row + c < P.S;
        l[j] = ok ? -P.lse[first + c] * log2e : -INFINITY;
        d[j] = ok ? -P.delta[first + c] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        out[j * 32 + lane] = l[j];
        out[BQ + j * 32 + lane] = d[j];
      }
      mbar_arrive(&bars->stat_full[it & 1]);
    };
    if (elect_one()) {
      mbar_expect_tx(&bars->kv_full, 2 * TILE);
      for (int c = 0; c < CHUNKS; ++c) {
        tma_load_2d(sK + c * CHUNK_BYTES, &tmap_k, &bars->kv_full, kv_head * D + c * 64, kv_row0);
        tma_load_2d(sV + c * CHUNK_BYTES, &tmap_v, &bars->kv_full, kv_head * D + c * 64, kv_row0);
      }
    }
    __syncwarp();
    load_q(0);
    load_do(0);
    if (iters > 1) load_q(1);
    load_stats(0);
    if (iters > 1) load_stats(1);
    for (int it = 1; it < iters && !__any_sync(0xffffffffu, *abort_flag != 0); ++it) {
      // dO is released after the dV product, Q after the dK product (the table's stage with it: dS is complete)
      if (!mbar_wait_warp(&bars->do_empty, (it - 1) & 1)) {
        if (lane == 0) { *abort_flag = 1; atomicCAS(P.err, 0, 401); }
        break;
      }
      if (lane == 0) stamp(0, 0, it);
      load_do(it);
      if (it + 1 == iters) break;
      if (!mbar_wait_warp(&bars->q_empty[(it + 1) & 1], ((it - 1) >> 1) & 1)) {
        if (lane == 0) { *abort_flag = 1; atomicCAS(P.err, 0, 413); }
        break;
      }
      if (lane == 0) stamp(0, 1, it);
      load_q(it + 1);
      load_stats(it + 1);
    }
  } else if (warp == 1) {
    // The whole warp runs this loop and an elected lane issues (warp-uniform control flow around
    // the tensor instructions costs the issuer less, and what it spends between two products is
    // time the pipe stands still; csrc/kernels/mma_probe.cu).
    constexpr int AB = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t id_s = make_idesc_f16(AB, 0, 0, BQ, BKV);     // K-major x K-major
    constexpr uint32_t id_q = make_idesc_f16(AB, 1, 1, BQ, D);       // MN-major x MN-major
    constexpr uint32_t id_t = make_idesc_f16(AB, 0, 1, BKV, D);      // K-major (or tensor memory) x MN-major
    // descriptor halves of the tiles, prepared once: an instruction then costs two integer adds
    constexpr uint32_t dhi = smem_desc_hi(1024);
    const uint32_t q_k = smem_desc_lo(smem_u32(sQ), 16), k_k = smem_desc_lo(smem_u32(sK), 16),
                   do_k = smem_desc_lo(smem_u32(sdO), 16), v_k = smem_desc_lo(smem_u32(sV), 16),
                   ds_k = smem_desc_lo(smem_u32(sdS), 16);
    const uint32_t do_m = smem_desc_lo(smem_u32(sdO), CHUNK_BYTES), ds_m = smem_desc_lo(smem_u32(sdS), CHUNK_BYTES),
                   q_m = smem_desc_lo(smem_u32(sQ), CHUNK_BYTES), k_m = smem_desc_lo(smem_u32(sK), CHUNK_BYTES);
    auto desc = [&](uint32_t lo, uint32_t off_bytes) { return smem_desc_join(lo + (off_bytes >> 4), dhi); };
    bool ok = true;
    auto fail = [&](int code) { if (lane == 0) atomicCAS(P.err, 0, code); ok = false; };
    auto mstamp = [&](int site, int it) { if (TRACE && lane == 0) stamp(1, site, it); };
    // S^T = K Q^T
    auto s_product = [&](int it) {
      const uint32_t q = q_k + (it & 1) * (TILE >> 4);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * CHUNK_BYTES + (kk % 4) * 32;
          umma_f16(tm_s, desc(k_k, off), desc(q, off), id_s, kk != 0);
        }
        umma_commit(&bars->s_full);
      }
      __syncwarp();
    };
    // dP^T = V dO^T
    auto dp_product = [&] {
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * CHUNK_BYTES + (kk % 4) * 32;
          umma_f16(tm_dp, desc(v_k, off), desc(do_k, off), id_s, kk != 0);
        }
        umma_commit(&bars->dp_full);
      }
      __syncwarp();
    };
    if (!mbar_wait_warp(&bars->kv_full, 0)) fail(402);
    if (ok && !mbar_wait_warp(&bars->q_full[0], 0)) fail(403);
    if (ok) {
      tc_fence_after();
      s_product(0);
      if (!mbar_wait_warp(&bars->do_full, 0)) fail(414);
    }
    if (ok) dp_product();
    for (int it = 0; it < iters && ok && !__any_sync(0xffffffffu, *abort_flag != 0); ++it) {
      const uint32_t ph = it & 1;
      const bool more = it + 1 < iters;
      mstamp(0, it);
      if (!mbar_wait_warp(&bars->p_full, ph)) { fail(405); break; }
      mstamp(1, it);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)         // reduction over the 128 query rows; P^T lies in 32-column pieces
          umma_f16_ts(tm_dv, tm_s + (kk / 2) * 32 + (kk % 2) * 8, desc(do_m, kk * 2048), id_t, (it | kk) != 0);
        umma_commit(&bars->do_empty);
      }
      __syncwarp();
      mstamp(2, it);
      if (more) {
        if (!mbar_wait_warp(&bars->q_full[(it + 1) & 1], ((it + 1) >> 1) & 1)) { fail(403); break; }
        // Over P^T, once dV has read it: an order is promised to products of one accumulator and shape only.  Without the wait
        // 0.4 % less (median of 56 shapes).
        if (!mbar_wait_warp(&bars->do_empty, ph)) { fail(418); break; }
        tc_fence_after();
        s_product(it + 1);
      }
      mstamp(3, it);
      if (!mbar_wait_warp(&bars->ds_full, ph)) { fail(409); break; }
      mstamp(4, it);
      tc_fence_after();
      if (elect_one()) {
        const uint32_t q = q_m + (it & 1) * (TILE >> 4);
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)         // reduction over the 128 query rows
          umma_f16(tm_dk, desc(ds_k, (kk / 4) * CHUNK_BYTES + (kk % 4) * 32), desc(q, kk * 2048), id_t, (it | kk) != 0);
        umma_commit(&bars->q_empty[it & 1]);
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk)        // reduction over the 128 kv rows
          umma_f16(tm_dq, desc(ds_m, kk * 2048), desc(k_m, kk * 2048), id_q, kk != 0);
        umma_commit(&bars->dq_full);
      }
      __syncwarp();
      mstamp(5, it);
      if (more && !mbar_wait_warp(&bars->do_full, (it + 1) & 1)) { fail(414); break; }
      mstamp(6, it);
      if (more) {
        if (!mbar_wait_warp(&bars->dq_read, ph)) { fail(404); break; }
        tc_fence_after();
        dp_product();
      }
      mstamp(7, it);
    }
    if (ok) {
      if (elect_one()) umma_commit(&bars->acc_full);
      __syncwarp();
    } else {
      *abort_flag = 1;
    }
    if (lane == 0) allow_next_kernel();              // this CTA's last product is under way
  } else if (warp == 2 + 4 * SPLIT) {
    // ------------------------------------------------------------ dQ store warp
    if (lane == 0) {
      for (int it = 0; it < iters && !*abort_flag; ++it) {
        const int head = head0 + it / q_blocks;
        const int m = nb + it % q_blocks;
        if (!mbar_wait(&bars->dqs_full, it & 1)) { *abort_flag = 1; atomicCAS(P.err, 0, 411); break; }
        stamp(4, 0, it);
        // the slabs inside the dS tile first: the next dS waits for them to be read
#pragma unroll
        for (int c = OWN_SLABS; c < D / 32; ++c)
          tma_reduce_add_2d(&tmap_dq, slab_ptr(c), head * D + c * 32, batch * P.S + m * BQ);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
#pragma unroll
        for (int c = 0; c < OWN_SLABS && c < D / 32; ++c)
          tma_reduce_add_2d(&tmap_dq, slab_ptr(c), head * D + c * 32, batch * P.S + m * BQ);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        stamp(4, 1, it);
        mbar_arrive(&bars->shared_free);
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        stamp(4, 2, it);
        mbar_arrive(&bars->own_free);
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  } else {
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;                // which part of the columns this warp owns
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint64_t scale2 = pm::pack2(P.scale_log2, P.scale_log2);
    constexpr int NC = BKV / (32 * SPLIT);           // 32-column chunks of S / dP per warp
    static_assert(NC >= 1, "at most four parts of 32 columns");
    // 32-column chunks of dQ / dK / dV per warp; with fewer chunks than parts the last parts have none
    constexpr int DC = (D / 32 >= SPLIT) ? (D / 32) / SPLIT : 1;
    const bool owns_d = part * DC < D / 32;
    bool ok = true;
    // the first and the last softmax warp record the timeline
    const int trole = (lane == 0 && warp == 2) ? 2 : ((lane == 0 && warp == 1 + 4 * SPLIT) ? 3 : -1);
    auto sstamp = [&](int site, int it) { if (TRACE && trole >= 0) stamp(trole, site, it); };
    // dQ of step `it` -> fp32 staging (32-column slabs of [128 rows][128 B], 128B-swizzled); rows
    // past the end of the sequence hold exact zeros (their P and dS are zero)
    auto dq_out = [&](int it) {
      if (!mbar_wait(&bars->dq_full, it & 1)) { atomicCAS(P.err, 0, 407); return false; }
      sstamp(6, it);
      tc_fence_after();
      if (owns_d) {                                  // uniform per warp
        uint32_t v[DC][32];
#pragma unroll
        for (int cc = 0; cc < DC; ++cc) tmem_ld_32x32(tm_dq + lane_addr + (part * DC + cc) * 32, v[cc]);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(&bars->dq_read);                 // the columns may be overwritten
        sstamp(7, it);
        if (it > 0 && !mbar_wait(&bars->own_free, (it - 1) & 1)) { atomicCAS(P.err, 0, 415); return false; }
#pragma unroll
        for (int cc = 0; cc < DC; ++cc) {
          uint8_t* slab = slab_ptr(part * DC + cc);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<uint4*>(slab + swz(r, u)) =
                make_uint4(v[cc][u * 4], v[cc][u * 4 + 1], v[cc][u * 4 + 2], v[cc][u * 4 + 3]);
        }
      } else {
        tc_fence_before();
        mbar_arrive(&bars->dq_read);
      }
      fence_proxy_async();
      mbar_arrive(&bars->dqs_full);
      sstamp(8, it);
      return true;
    };
    for (int it = 0; it < iters; ++it) {
      const uint32_t ph = it & 1;
      const bool diag = it % q_blocks == 0;          // the block on the diagonal
      const float* stat = sStat + (it & 1) * 2 * BQ + part * NC * 32;
      float p[NC][32];
      sstamp(0, it);
      // ---- P as soon as S is complete
      if (!mbar_wait(&bars->stat_full[it & 1], (it >> 1) & 1)) { atomicCAS(P.err, 0, 417); ok = false; break; }
      if (!mbar_wait(&bars->s_full, ph)) { atomicCAS(P.err, 0, 406); ok = false; break; }
      sstamp(1, it);
      tc_fence_after();
      {
        uint32_t sv[NC][32];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) tmem_ld_32x32(tm_s + lane_addr + (part * NC + cc) * 32, sv[cc]);
        tmem_ld_wait();
        sstamp(2, it);
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          const int c = part * NC + cc;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 l = *reinterpret_cast<const float4*>(stat + cc * 32 + i);
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
              float a, b;
              pm::unpack2(pm::fma2(pm::pack2(__uint_as_float(sv[cc][i + h]), __uint_as_float(sv[cc][i + h + 1])), scale2,
                                   h ? pm::pack2(l.z, l.w) : pm::pack2(l.x, l.y)), a, b);
              if ((POLY >> (((i + h) >> 1) & 7)) & 1u) {
                pm::ex2_poly2(a, b, p[cc][i + h], p[cc][i + h + 1]);
              } else {
                p[cc][i + h] = pm::ex2(a);
                p[cc][i + h + 1] = pm::ex2(b);
              }
            }
          }
          if (diag) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i < r) p[cc][i] = 0.f;    // the query comes before the key
          }
          // P^T over the first half of this warp's own columns of S^T
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = pm::cvt2<T>(p[cc][2 * i], p[cc][2 * i + 1]);
          tmem_st_32x16(tm_s + lane_addr + c * 32, w);
        }
        tmem_st_wait();
      }
      tc_fence_before();
      mbar_arrive(&bars->p_full);
      sstamp(3, it);
      // ---- the step before this one's dQ, computed meanwhile
      if (it > 0 && !dq_out(it - 1)) { ok = false; break; }
      // ---- dS once dP is complete
      if (!mbar_wait(&bars->dp_full, ph)) { atomicCAS(P.err, 0, 410); ok = false; break; }
      sstamp(4, it);
      // part of the previous dQ tile left through the dS tile: its reduce-add must have read it
      if (it > 0 && !mbar_wait(&bars->shared_free, (it - 1) & 1)) { atomicCAS(P.err, 0, 412); ok = false; break; }
      sstamp(5, it);
      tc_fence_after();
      {
        uint32_t dv[NC][32];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) tmem_ld_32x32(tm_dp + lane_addr + (part * NC + cc) * 32, dv[cc]);
        tmem_ld_wait();
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          const int c = part * NC + cc;
          uint8_t* dc = sdS + (c / 2) * CHUNK_BYTES;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t w[4];
#pragma unroll
            for (int h4 = 0; h4 < 2; ++h4) {
              const int i = u * 8 + h4 * 4;
              const float4 d = *reinterpret_cast<const float4*>(stat + BQ + cc * 32 + i);
              float a, b;
              pm::unpack2(pm::mul2(pm::add2(pm::pack2(__uint_as_float(dv[cc][i]), __uint_as_float(dv[cc][i + 1])),
                                            pm::pack2(d.x, d.y)), pm::pack2(p[cc][i], p[cc][i + 1])), a, b);
              w[2 * h4] = pm::cvt2<T>(a, b);
              pm::unpack2(pm::mul2(pm::add2(pm::pack2(__uint_as_float(dv[cc][i + 2]), __uint_as_float(dv[cc][i + 3])),
                                            pm::pack2(d.z, d.w)), pm::pack2(p[cc][i + 2], p[cc][i + 3])), a, b);
              w[2 * h4 + 1] = pm::cvt2<T>(a, b);
            }
            *reinterpret_cast<uint4*>(dc + swz(r, (c % 2) * 4 + u)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      tc_fence_before();
      fence_proxy_async();
      mbar_arrive(&bars->ds_full);
      sstamp(9, it);
    }
    if (ok && !dq_out(iters - 1)) ok = false;
    if (ok && !mbar_wait(&bars->acc_full, 0)) { atomicCAS(P.err, 0, 408); ok = false; }
    if (ok) {
      tc_fence_after();
      const int kv_pos = nb * BKV + r;
      // every lane of a warp issues the same tensor-memory loads (they are warp-wide
      // instructions); only the stores depend on whether the lane's row exists
      const bool row_ok = kv_pos < P.S;
      const int64_t row = (int64_t)(batch * P.S + (row_ok ? kv_pos : 0));
      T* dk_row = reinterpret_cast<T*>(P.dk) + row * P.dk_stride + kv_head * D;
      T* dv_row = reinterpret_cast<T*>(P.dv) + row * P.dv_stride + kv_head * D;
      // more than one part (nothing of this is kept through the walk: the kernel has no register to spare)
      const int64_t plane = (int64_t)P.B * P.S * P.Hkv * D;
      const int part_id = (head0 - kv_head * group) / P.part_heads;
      float* dk_part = P.kv_part + 2 * part_id * plane + (row * P.Hkv + kv_head) * D;
#pragma unroll 1
      for (int c = part * DC; owns_d && c < (part + 1) * DC; ++c) {
        uint32_t a[32], b[32];
        tmem_ld_32x32(tm_dk + lane_addr + c * 32, a);
        tmem_ld_32x32(tm_dv + lane_addr + c * 32, b);
        tmem_ld_wait();
        if (row_ok && P.splits > 1) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            reinterpret_cast<uint4*>(dk_part + c * 32)[u] = make_uint4(a[u * 4], a[u * 4 + 1], a[u * 4 + 2], a[u * 4 + 3]);
            reinterpret_cast<uint4*>(dk_part + plane + c * 32)[u] =
                make_uint4(b[u * 4], b[u * 4 + 1], b[u * 4 + 2], b[u * 4 + 3]);
          }
        } else if (row_ok) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float t[8], w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              t[i] = __uint_as_float(a[u * 8 + i]) * P.scale;          // dS carried no softmax scale
              w[i] = __uint_as_float(b[u * 8 + i]);
            }
            *reinterpret_cast<uint4*>(dk_row + c * 32 + u * 8) = pack8<T>(t);
            *reinterpret_cast<uint4*>(dv_row + c * 32 + u * 8) = pack8<T>(w);
          }
        }
      }
    } else {
      *abort_flag = 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// delta[b,h,s] = sum_d dO * O.  D / 8 lanes per (head, token) row (16 bytes of each tensor per
// lane), so a warp covers 32 * 8 / D rows at once, and every thread does that for two rows with
// all four loads in flight.  Rows are numbered in the order of delta ([b, h, s]), so neighbouring
// lanes write neighbouring floats; the reads are whole 2 * D-byte pieces either way.  The rows of
// dq_acc, which the backward adds into, are zeroed on the way (a memset of its own would also stand
// between this kernel and the one before it).  D in {64, 128}.
constexpr int kDeltaRowsPerBlock(int D) { return 2 * 8 * (256 / D); }   // 2 passes x 8 warps x rows per warp

template <typename T>
__global__ void __launch_bounds__(256) attn_delta_kernel(const T* o, const T* d_o, int64_t do_stride,
                                                         float* delta, float* dq_acc, int B, int S, int Hq,
                                                         int D) {
  wait_previous_kernel();
  const int lpr = D / 8, rpw = 32 / lpr;             // lanes per row, rows per warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane % lpr;
  const int64_t rows = (int64_t)B * S * Hq;
  const int64_t row0 = (int64_t)blockIdx.x * (2 * 8 * rpw) + warp * rpw + lane / lpr;
  float acc[2];
  uint4 a[2], b[2];
  bool ok[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int64_t row = row0 + (int64_t)p * 8 * rpw;
    ok[p] = row < rows;
    const int64_t r = ok[p] ? row : 0;
    const int64_t bh = r / S;
    const int64_t tok = (bh / Hq) * S + r % S;
    const int h = (int)(bh % Hq);
    a[p] = *reinterpret_cast<const uint4*>(o + (tok * Hq + h) * D + sub * 8);
    b[p] = *reinterpret_cast<const uint4*>(d_o + tok * do_stride + (int64_t)h * D + sub * 8);
    if (ok[p]) {
      uint4* z = reinterpret_cast<uint4*>(dq_acc + (tok * Hq + h) * D + sub * 8);
      z[0] = z[1] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  allow_next_kernel();
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float x[8], y[8];
    unpack8<T>(a[p], x);
    unpack8<T>(b[p], y);
    acc[p] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[p] += x[k] * y[k];
    for (int off = lpr / 2; off > 0; off >>= 1) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], off);
    const int64_t row = row0 + (int64_t)p * 8 * rpw;
    if (ok[p] && sub == 0) delta[row] = acc[p];
  }
}

// dq (16-bit, token stride) <- scale * dq_acc (fp32, contiguous [tokens, W])
template <typename T>
__global__ void __launch_bounds__(256) attn_dq_cast_kernel(const float* acc, T* dq,
                                                           int64_t dq_stride, int64_t tokens, int W,
                                                           float scale) {
  wait_previous_kernel();
  const int vec = W / 8;
  const int64_t total = tokens * vec;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / vec;
    const int c = (int)(idx % vec) * 8;
    const float4 a = *reinterpret_cast<const float4*>(acc + t * W + c);
    const float4 b = *reinterpret_cast<const float4*>(acc + t * W + c + 4);
    float v[8] = {a.x * scale, a.y * scale, a.z * scale, a.w * scale,
                  b.x * scale, b.y * scale, b.z * scale, b.w * scale};
    *reinterpret_cast<uint4*>(dq + t * dq_stride + c) = pack8<T>(v);
  }
  allow_next_kernel();
}

// dk, dv (16-bit, token strides) <- the sums over `splits` parts of kv_part (see BwdParams), dk times
// the softmax scale.  blockIdx.y: 0 dk, 1 dv.  W = Hkv * D columns.
template <typename T>
__global__ void __launch_bounds__(256) attn_dkv_sum_kernel(const float* kv_part, int splits, T* dk,
                                                           int64_t dk_stride, T* dv, int64_t dv_stride,
                                                           int64_t tokens, int W, float scale) {
  wait_previous_kernel();
  const int vec = W / 8;
  const int64_t total = tokens * vec, plane = tokens * W;
  const float* src = kv_part + blockIdx.y * plane;
  T* out = blockIdx.y ? dv : dk;
  const int64_t stride = blockIdx.y ? dv_stride : dk_stride;
  const float f = blockIdx.y ? 1.f : scale;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / vec;
    const int c = (int)(idx % vec) * 8;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
#pragma unroll 4
    for (int p = 0; p < splits; ++p) {
      const float4* q = reinterpret_cast<const float4*>(src + 2 * p * plane + t * W + c);
      const float4 a = q[0], b = q[1];
      v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
      v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= f;
    *reinterpret_cast<uint4*>(out + t * stride + c) = pack8<T>(v);
  }
  allow_next_kernel();
}

}  // namespace attn
}  // namespace ft
