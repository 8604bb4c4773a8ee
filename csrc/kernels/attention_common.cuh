// Definitions shared by the causal flash-attention kernels (attention_fwd2.cuh,
// attention_bwd.cuh): tile sizes, the forward parameter block and the
// 128-byte swizzle of a [rows][64] shared-memory chunk.
#pragma once
#include "common.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"

namespace ft {
namespace attn {

using namespace ft::sm100;

constexpr int BQ = 128, BKV = 128, KV_STAGES = 2;

// Order of the CTAs of a causal grid: (head, block) jobs whose cost grows with the number of blocks on
// the other side of the diagonal, handed to the SMs in the order of blockIdx.  Heads are taken
// `chunk` at a time and inside a chunk the heaviest block of every head comes first, then the next
// lighter one of every head (longest job first), so that what the last SMs still work on are short
// jobs.  Walking head by head instead (each head's blocks from heavy to light) left the last heads'
// heavy jobs to the end.  Measured, walking by head -> by weight: forward 32 heads x 4096 tokens 184 ->
// 155 us (list scheduling on 148 SMs says 83 -> 64 units), backward of 16 (batch, kv head) groups of 8
// query heads x 4096 1789 -> 1517 us (607 -> 485).  A chunk's keys and values (forward) or queries and
// output gradients (backward) stay within about half of L2, because its jobs run side by side.
struct CausalJob { int head, rank; };                // rank 0: the heaviest block of the head

__device__ __forceinline__ CausalJob causal_job(int idx, int heads, int blocks, int chunk) {
  const int c = idx / (chunk * blocks);
  const int first = c * chunk;
  const int n = min(chunk, heads - first);
  const int r = idx - c * chunk * blocks;
  return {first + r % n, r / n};
}

// heads per chunk for a working set of `bytes` per head: chunks of equal size and at least two heads.  A
// minimum of 16 (so that a chunk's jobs are many for 148 SMs) let long contexts run out of L2: backward, walking by
// head / 16 / 2: 1 x 16384, 16 heads of 64 2239 / 2302 / 2148 us, 1 x 32768, 8 of 128 6165 / 6351 / 6137, 1 x 65536,
// 8 of 64 17263 / 18002 / 16968; up to 8192 tokens 2 and 16 are the same.  All heads in one chunk: 8 x 4096, 40 of
// 128 6245 us instead of 4860.
inline int causal_chunk(int64_t heads, int64_t bytes) {
  int64_t c = (64LL << 20) / (bytes > 0 ? bytes : 1);
  if (c < 2) c = 2;
  if (c > heads) c = heads;
  const int64_t chunks = (heads + c - 1) / c;
  return (int)((heads + chunks - 1) / chunks);
}

struct FwdParams {
  void* o;                 // [B, S, Hq, D] contiguous
  float* lse;              // [B, Hq, S]: natural log of sum exp(scale * s) per query row
  int B, S, Hq, Hkv;
  int chunk;               // heads per chunk of the CTA order (causal_job)
  float scale_log2;        // softmax scale * log2(e)
  float scale_ln;          // softmax scale
  int q_col0, k_col0, v_col0;   // column of head 0 inside the respective tensor map rows
  int* err;
  // timeline capture (TRACE instantiation only): clock64() of CTA trace_cta at the hand-over points
  // of K/V blocks trace_it0 .. trace_it0 + 7, as trace[(role * 8 + site) * 8 + block]
  long long* trace;
  int trace_cta, trace_it0;
};

// byte offset of 16-byte unit `u` (0..7) of row `r` inside a 128B-swizzled [rows][64] chunk
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t u) {
  return (r >> 3) * 1024 + (r & 7) * 128 + ((u ^ (r & 7)) << 4);
}

}  // namespace attn
}  // namespace ft
