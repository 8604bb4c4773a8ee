// Host launchers of the causal flash-attention kernels (attention_fwd*.cuh,
// attention_bwd*.cuh).  q / k / v may be views into one packed QKV tensor: each is
// described by its own base pointer and token stride, rows of H*D columns.
// Replaces the scaled-dot-product attention library call a PyTorch model makes.
#include <algorithm>

#include <cstdlib>

#include "attention_bwd.cuh"
#include "attention_fwd2.cuh"
#include "gemm_host.h"

namespace {

using namespace ft;
using namespace ft::attn;

// dynamic shared memory a CTA may ask for on sm_100 (227 KB)
constexpr int kMaxDynamicSmem = 232448;
static_assert(Fwd2Smem<128, 2>::BYTES <= kMaxDynamicSmem && BwdSmem<128>::BYTES <= kMaxDynamicSmem,
              "an attention kernel outgrew the shared memory of an SM");

// bytes of Q (and of O, dO or the 16-bit dQ)
template <typename Params>
int64_t query_bytes(const Params& P, int D) { return (int64_t)P.B * P.S * P.Hq * D * 2; }

// Query tiles of a CTA in the forward, for `heads` (batch, query head)s of `tiles` tiles: the number with the shorter expected time, in clocks.
// Pairs: every SM takes the next job when it is done with one, heaviest first; a K/V block takes a pair 3 365, a job 7 000 besides
// and the launch 3 000.  Single tiles of 64-wide heads, two CTAs an SM: 2 700 a block at least, 2 312 of an SM's time where two share it,
// 9 000 for the first and 5 000 for what comes behind the first two of an SM.  Pairs, singles, us: 24 heads of 512 tokens 11.7 and 9.2,
// of 1024 18.3 and 15.5; 75 of 1000 33.1 and 27.2, 48 of 1000 18.9 and 19.8; 8 of 2048 30.5 and 25.0.  Longer sequences have work
// to share out in pairs: 16 heads of 4096 58.5 and 66.6, 4 of 16384 217 and 234 (16 of 8192 211 and 205).
constexpr int kFwdSingleTiles = 16;
int fwd_tiles(int64_t heads, int tiles, int D) {
  if (D != 64 || tiles > kFwdSingleTiles) return 2;
  constexpr int SMS = 148;
  const double total = (double)heads * tiles * (tiles + 1) / 2, jobs = (double)heads * tiles;
  const double singles = 9000 + std::max(2700.0 * tiles, total / SMS * 2312) + (jobs > 2 * SMS ? 5000 * (jobs - 2 * SMS) / (2 * SMS) : 0);
  if (total > 2000 * SMS) return 2;                  // whole rounds by far: as good either way, and the walk below is long
  // SMs by the time at which they are free, soonest first; a rank's jobs are alike
  struct Free { double at; int64_t n; } sm[kFwdSingleTiles + 2] = {{0, SMS}};
  int count = 1;
  double pairs = 0;
  for (int last = tiles; last > 0; last -= last % 2 ? 1 : 2) {      // K/V blocks of the pair: those of its last tile
    const double length = 3365.0 * last + 7000;
    for (int64_t left = heads; left > 0;) {
      const Free f = sm[0];
      const int64_t n = left < f.n ? left : f.n;
      left -= n;
      int i = 0;
      if (n == f.n) for (--count; i < count; ++i) sm[i] = sm[i + 1];
      else sm[0].n -= n;
      const double end = f.at + length;
      pairs = std::max(pairs, end);
      if (count > kFwdSingleTiles) return 2;
      for (i = count; i > 0 && sm[i - 1].at > end; --i) sm[i] = sm[i - 1];
      if (i > 0 && sm[i - 1].at == end) {            // moved one too far: close the gap again
        sm[i - 1].n += n;
        for (; i < count; ++i) sm[i] = sm[i + 1];
      } else {
        sm[i] = {end, n};
        ++count;
      }
    }
  }
  return singles < pairs + 3000 ? 1 : 2;
}

// Forward: one CTA per pair of query blocks, or per block.
template <typename T, int D, bool TRACE, int TILES>
int launch_fwd2_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& P,
                  cudaStream_t s) {
  constexpr int BYTES = Fwd2Smem<D, TILES>::BYTES;
  auto kern = attn_fwd2_kernel<T, D, 0x00u, TRACE, TILES>;
  static DynamicSmem smem;
  smem.grant(kern, BYTES);
  const int num_jobs = ((P.S + BQ - 1) / BQ + TILES - 1) / TILES;
  launch_overlapped(kern, P.B * P.Hq * num_jobs, f2_threads(TILES), BYTES, s, 1,
                    overlap_bytes(query_bytes(P, D) * 2), tq, tk, tv, P);
  return 0;
}

// The timeline instantiations exist for bf16 at head size 128 only (the benchmark shapes).
template <typename T, int D>
int launch_fwd2(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& P,
                cudaStream_t s) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value && D == 128) {
    if (P.trace != nullptr) return launch_fwd2_t<T, D, true, 2>(tq, tk, tv, P, s);
  }
  if constexpr (D == 64) {
    if (fwd_tiles((int64_t)P.B * P.Hq, (P.S + BQ - 1) / BQ, D) == 1) return launch_fwd2_t<T, D, false, 1>(tq, tk, tv, P, s);
  }
  return launch_fwd2_t<T, D, false, 2>(tq, tk, tv, P, s);
}

// Backward: four threads per score row (2.6 % faster than two at the 13B shape, 96 registers
// instead of 158); every other pair of probabilities takes the polynomial 2^x (4.524 ms against
// 4.752 ms with none and 4.635 ms with five of eight at the 13B shape).
constexpr int kBwdSplit = 4;

template <typename T, int D, bool TRACE>
int launch_bwd_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                 const CUtensorMap& tdq, const BwdParams& P, cudaStream_t s) {
  auto kern = attn_bwd_kernel<T, D, kBwdSplit, TRACE>;
  static DynamicSmem smem;
  smem.grant(kern, BwdSmem<D>::BYTES);
  const int num_blk = (P.S + BQ - 1) / BQ;
  launch_overlapped(kern, P.B * P.Hkv * P.splits * num_blk, bwd_threads(kBwdSplit), BwdSmem<D>::BYTES, s, 1,
                    overlap_bytes(query_bytes(P, D) * 2), tq, tk, tv, tdo, tdq, P);
  return 0;
}

template <typename T, int D>
int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
               const CUtensorMap& tdq, const BwdParams& P, cudaStream_t s) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value && D == 128) {
    if (P.trace != nullptr) return launch_bwd_t<T, D, true>(tq, tk, tv, tdo, tdq, P, s);
  }
  return launch_bwd_t<T, D, false>(tq, tk, tv, tdo, tdq, P, s);
}

template <typename T>
void launch_pre_post(bool post, const void* o, const void* d_o, int64_t do_stride, float* delta,
                     float* dq_acc, void* dq, int64_t dq_stride, int B, int S, int Hq, int D,
                     float scale, cudaStream_t s) {
  if (!post) {
    const int64_t rows = (int64_t)B * S * Hq;
    const int per_block = kDeltaRowsPerBlock(D);
    launch_overlapped(attn_delta_kernel<T>, (unsigned)((rows + per_block - 1) / per_block), 256, 0, s, 1,
        overlap_bytes(rows * D * 8), (const T*)o, (const T*)d_o, do_stride, delta, dq_acc, B, S, Hq, D);
  } else {
    const int64_t tokens = (int64_t)B * S;
    launch_overlapped(attn_dq_cast_kernel<T>, grid_for(tokens * (Hq * D / 8), 256), 256, 0, s, 1,
                      overlap_bytes(tokens * Hq * D * 6), dq_acc, (T*)dq, dq_stride,
                                                                                tokens, Hq * D, scale);
  }
}

template <typename T>
void launch_dkv_sum(const BwdParams& P, int D, cudaStream_t s) {
  const int64_t tokens = (int64_t)P.B * P.S;
  const int W = P.Hkv * D;
  launch_overlapped(attn_dkv_sum_kernel<T>, dim3(grid_for(tokens * (W / 8), 256), 2), 256, 0, s, 1,
      overlap_bytes(tokens * W * 8 * P.splits), P.kv_part, P.splits, (T*)P.dk, P.dk_stride, (T*)P.dv, P.dv_stride, tokens, W, P.scale);
}

}  // namespace

extern "C" {

// o[B,S,Hq,D], lse[B,Hq,S] <- causal attention of q[B,S,Hq,D], k/v[B,S,Hkv,D].
// *_stride: elements between consecutive tokens of that tensor.  D in {64, 128}.
// ft_attn_fwd_traced additionally records the timeline of one CTA: `trace` is nullptr or a device
// buffer of 3 * 8 * 8 clock values (see FwdParams).
int ft_attn_fwd_traced(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                       int64_t v_stride, void* o, float* lse, int B, int S, int Hq, int Hkv, int D,
                       float scale, int dtype, cudaStream_t stream, long long* trace, int trace_cta,
                       int trace_it0) {
  if (D != 64 && D != 128) return -1;
  if (dtype != kBF16 && dtype != kF16) return -2;
  if (Hq % Hkv) return -3;
  int dev = 0;
  cudaGetDevice(&dev);
  CUtensorMap tq, tk, tv;
  int rc = gemm::make_tmap(&tq, q, (uint64_t)Hq * D, (uint64_t)B * S, (uint64_t)q_stride, 64, BQ, dtype);
  if (rc) return rc;
  rc = gemm::make_tmap(&tk, k, (uint64_t)Hkv * D, (uint64_t)B * S, (uint64_t)k_stride, 64, BKV, dtype);
  if (rc) return rc;
  rc = gemm::make_tmap(&tv, v, (uint64_t)Hkv * D, (uint64_t)B * S, (uint64_t)v_stride, 64, BKV, dtype);
  if (rc) return rc;
  FwdParams P;
  P.o = o; P.lse = lse; P.B = B; P.S = S; P.Hq = Hq; P.Hkv = Hkv;
  // K and V of a kv head, shared by its query heads
  P.chunk = causal_chunk((int64_t)B * Hq, (int64_t)S * D * 4 / (Hq / Hkv));
  P.scale_log2 = scale * 1.4426950408889634f;
  P.scale_ln = scale;
  P.q_col0 = P.k_col0 = P.v_col0 = 0;
  P.err = gemm::error_word(dev);
  P.trace = trace; P.trace_cta = trace_cta; P.trace_it0 = trace_it0;
  if (dtype == kBF16) {
    if (D == 128) launch_fwd2<__nv_bfloat16, 128>(tq, tk, tv, P, stream);
    else launch_fwd2<__nv_bfloat16, 64>(tq, tk, tv, P, stream);
  } else {
    if (D == 128) launch_fwd2<__half, 128>(tq, tk, tv, P, stream);
    else launch_fwd2<__half, 64>(tq, tk, tv, P, stream);
  }
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_attn_fwd(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                int64_t v_stride, void* o, float* lse, int B, int S, int Hq, int Hkv, int D, float scale,
                int dtype, cudaStream_t stream) {
  return ft_attn_fwd_traced(q, q_stride, k, k_stride, v, v_stride, o, lse, B, S, Hq, Hkv, D, scale, dtype,
                            stream, nullptr, 0, 0);
}

// Query tiles of a CTA in the forward of `heads` (batch, query head)s over S tokens (the rule, for its tests).
int ft_attn_fwd_tiles(int64_t heads, int S, int D) { return fwd_tiles(heads, (S + BQ - 1) / BQ, D); }

// Over how many CTAs the query heads of one kv head are at most divided in the backward; ft_attn_bwd_parts
// chooses.  A CTA walks all the query blocks at or below its kv block for each of its heads, so with few
// (batch, kv head) groups the longest job outlasts everybody else's work: 8 groups of 8 heads over 2048 tokens
// are 128 jobs of up to 128 blocks where 60 per SM would do, one group of 32 heads over 1024 tokens keeps 8 of
// 148 SMs busy.  Splits are added until the longest job, heads / splits x blocks, is no longer than an SM's even
// share of the total, heads x groups x blocks (blocks + 1) / 2 / 148; the partial sums take 16 bytes per split and
// element of K and are only written where there is more than one.
int ft_attn_bwd_splits(int B, int S, int Hq, int Hkv) {
  if (B <= 0 || S <= 0 || Hkv <= 0 || Hq % Hkv) return 1;
  const int64_t blocks = (S + BQ - 1) / BQ, share = (int64_t)B * Hkv * (blocks + 1);
  const int heads = Hq / Hkv;
  int64_t splits = (2 * 148 + share - 1) / share;
  if (splits > heads) splits = heads;
  const int64_t part = (heads + splits - 1) / splits;
  return (int)((heads + part - 1) / part);
}

// Into how many parts the backward divides the query heads of a kv head: of the divisions up to
// ft_attn_bwd_splits the one with the shortest expected time, in query blocks of one head (1.8 us for heads of
// 64, 2.7 us for 128).  A CTA costs 5 blocks besides its work; more CTAs than SMs run at the average load and half a
// CTA's cost more; several parts cost a kernel (1.5) and their partial sums (1 or 1.5 for a CTA on every SM).  Even
// loads alone are no reason to split: 40 groups of 4 heads of 64 over 256 tokens take 29.0 us whole and 34.0 us in two
// parts, 40 of 8 of 128 over 256 79.9 and 82.6.  Measured over 96 shapes of 2 to 8 heads, 2 to 64 groups and
// 1 to 32 blocks for each head size, every division timed: 0.08 % off the best division on average for heads of 64, 0.07 %
// for 128 (dividing up to ft_attn_bwd_splits 6.6 and 10.5 %, at worst 1.74x; never dividing 56 and 47 %), at worst 6 % (16
// groups of 2 of 64 over 1024 tokens, whole 41.0 us, halves 38.6), never more than 3.3 % behind the whole.
int ft_attn_bwd_parts(int B, int S, int Hq, int Hkv, int D) {
  const int most = ft_attn_bwd_splits(B, S, Hq, Hkv);
  if (most <= 1) return 1;
  const int64_t blocks = (S + BQ - 1) / BQ, groups = (int64_t)B * Hkv;
  const int heads = Hq / Hkv;
  const double total = 0.5 * groups * heads * blocks * (blocks + 1), fixed = 5;
  int best = 1;
  double least = 0;
  for (int n = 1; n <= most; ++n) {
    const int part = (heads + n - 1) / n;
    if ((n - 1) * part >= heads) continue;             // a part without a head
    const double jobs = (double)groups * n * blocks;
    double time = part * blocks + fixed;
    if (jobs > 148) time = std::max(time, (total + jobs * fixed) / 148 + fixed / 2);
    if (n > 1) time += 1.5 + (D == 128 ? 1.5 : 1.0) * jobs / 148;
    if (n == 1 || time < least) { best = n; least = time; }
  }
  return best;
}

// Gradients of ft_attn_fwd (ft_attn_bwd), optionally with a timeline of one CTA: `trace` is
// nullptr or a device buffer of 5 * 16 * 8 clock values (see BwdParams).  d_o is [B,S,Hq,D] with token
// stride do_stride; o and lse are the forward's outputs.  Scratch provided by the caller: delta
// [B*Hq*S] floats, dq_acc [B*S*Hq*D] floats (zeroed here) and, with `splits` (ft_attn_bwd_parts(...)) above 1, kv_part of splits * 2 * B*S*Hkv*D floats.  splits 1 (kv_part unused) is valid for every
// shape.  dq / dk / dv are written with their own token strides, so they may be views of one packed
// tensor.
int ft_attn_bwd_split(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                      int64_t v_stride, const void* o, const void* d_o, int64_t do_stride, const float* lse,
                      float* delta, float* dq_acc, float* kv_part, int splits, void* dq, int64_t dq_stride,
                      void* dk, int64_t dk_stride, void* dv, int64_t dv_stride, int B, int S, int Hq, int Hkv,
                      int D, float scale, int dtype, cudaStream_t stream, long long* trace, int trace_cta,
                      int trace_it0) {
  if (D != 64 && D != 128) return -1;
  if (dtype != kBF16 && dtype != kF16) return -2;
  if (Hq % Hkv) return -3;
  if (splits < 1 || splits > Hq / Hkv || (splits > 1 && kv_part == nullptr)) return -3;
  int dev = 0;
  cudaGetDevice(&dev);
  CUtensorMap tq, tk, tv, tdo;
  int rc = gemm::make_tmap(&tq, q, (uint64_t)Hq * D, (uint64_t)B * S, (uint64_t)q_stride, 64, BQ, dtype);
  if (rc) return rc;
  rc = gemm::make_tmap(&tk, k, (uint64_t)Hkv * D, (uint64_t)B * S, (uint64_t)k_stride, 64, BKV, dtype);
  if (rc) return rc;
  rc = gemm::make_tmap(&tv, v, (uint64_t)Hkv * D, (uint64_t)B * S, (uint64_t)v_stride, 64, BKV, dtype);
  if (rc) return rc;
  rc = gemm::make_tmap(&tdo, d_o, (uint64_t)Hq * D, (uint64_t)B * S, (uint64_t)do_stride, 64, BQ, dtype);
  if (rc) return rc;
  // dq_acc viewed as [B*S, Hq*D] fp32; the kernel adds 128-row x 32-column slabs into it
  CUtensorMap tdq;
  rc = gemm::make_tmap(&tdq, dq_acc, (uint64_t)Hq * D, (uint64_t)B * S, (uint64_t)Hq * D, 32, BQ, kF32);
  if (rc) return rc;
  BwdParams P;
  P.lse = lse; P.delta = delta; P.dq_acc = dq_acc;
  P.dk = dk; P.dk_stride = dk_stride; P.dv = dv; P.dv_stride = dv_stride;
  P.B = B; P.S = S; P.Hq = Hq; P.Hkv = Hkv;
  // Q, dO and the fp32 dQ of the query head a group works on; the jobs of a chunk walk their query
  // heads in the same order
  P.splits = splits;
  P.part_heads = (Hq / Hkv + splits - 1) / splits;
  if ((splits - 1) * P.part_heads >= Hq / Hkv) return -3;       // a part without a head
  P.kv_part = kv_part;
  P.chunk = causal_chunk((int64_t)B * Hkv * splits, (int64_t)S * D * 8);
  P.scale = scale; P.scale_log2 = scale * 1.4426950408889634f;
  P.err = gemm::error_word(dev);
  P.trace = trace; P.trace_cta = trace_cta; P.trace_it0 = trace_it0;
  if (dtype == kBF16) {
    launch_pre_post<__nv_bfloat16>(false, o, d_o, do_stride, delta, dq_acc, nullptr, 0, B, S, Hq, D, scale, stream);
    if (D == 128) launch_bwd<__nv_bfloat16, 128>(tq, tk, tv, tdo, tdq, P, stream);
    else launch_bwd<__nv_bfloat16, 64>(tq, tk, tv, tdo, tdq, P, stream);
    launch_pre_post<__nv_bfloat16>(true, nullptr, nullptr, 0, nullptr, dq_acc, dq, dq_stride, B, S, Hq, D, scale, stream);
    if (splits > 1) launch_dkv_sum<__nv_bfloat16>(P, D, stream);
  } else {
    launch_pre_post<__half>(false, o, d_o, do_stride, delta, dq_acc, nullptr, 0, B, S, Hq, D, scale, stream);
    if (D == 128) launch_bwd<__half, 128>(tq, tk, tv, tdo, tdq, P, stream);
    else launch_bwd<__half, 64>(tq, tk, tv, tdo, tdq, P, stream);
    launch_pre_post<__half>(true, nullptr, nullptr, 0, nullptr, dq_acc, dq, dq_stride, B, S, Hq, D, scale, stream);
    if (splits > 1) launch_dkv_sum<__half>(P, D, stream);
  }
  FT_LAUNCHED(splits > 1 ? 4 : 3);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_attn_bwd_traced(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                       int64_t v_stride, const void* o, const void* d_o, int64_t do_stride, const float* lse,
                       float* delta, float* dq_acc, void* dq, int64_t dq_stride, void* dk, int64_t dk_stride,
                       void* dv, int64_t dv_stride, int B, int S, int Hq, int Hkv, int D, float scale,
                       int dtype, cudaStream_t stream, long long* trace, int trace_cta, int trace_it0) {
  return ft_attn_bwd_split(q, q_stride, k, k_stride, v, v_stride, o, d_o, do_stride, lse, delta, dq_acc, nullptr, 1,
                           dq, dq_stride, dk, dk_stride, dv, dv_stride, B, S, Hq, Hkv, D, scale, dtype, stream, trace,
                           trace_cta, trace_it0);
}

int ft_attn_bwd(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                int64_t v_stride, const void* o, const void* d_o, int64_t do_stride, const float* lse,
                float* delta, float* dq_acc, void* dq, int64_t dq_stride, void* dk, int64_t dk_stride,
                void* dv, int64_t dv_stride, int B, int S, int Hq, int Hkv, int D, float scale, int dtype,
                cudaStream_t stream) {
  return ft_attn_bwd_traced(q, q_stride, k, k_stride, v, v_stride, o, d_o, do_stride, lse, delta, dq_acc, dq,
                            dq_stride, dk, dk_stride, dv, dv_stride, B, S, Hq, Hkv, D, scale, dtype, stream,
                            nullptr, 0, 0);
}

}  // extern "C"
