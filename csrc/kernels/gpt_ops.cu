// Bandwidth-bound ops of a GPT-style block (LayerNorm, biased projections, tanh
// GELU), bf16 / fp16 I/O with fp32 math, plus a register-resident RMSNorm built
// from the same row kernel.
//
//   ft_norm_fwd / ft_norm_bwd_into      LayerNorm (mean + rstd saved) or RMSNorm (rstd
//                                  saved).  A row is read ONCE: kept in registers
//                                  across the reductions (forward) or staged in a
//                                  shared-memory ring (backward), so nothing is
//                                  re-read from L2.
//   ft_bias_act_fwd / _bwd         y = act(x + bias), act in {identity, tanh GELU};
//                                  the backward writes dx and the per-CTA column
//                                  sums of dx (the bias gradient) in one pass.
//   ft_parts_reduce                sums the per-CTA partial rows into the parameter
//                                  gradient.
//
// The reference has no model code (its users bring Megatron-style GPT blocks whose
// fused bias-GELU and LayerNorm come from Megatron / Apex); these are the
// counterparts of those fused kernels.  Every pointer that is accessed through
// 128-bit vectors is checked for 16-byte alignment on the host; a launch that would
// be misaligned is refused with -2 instead of faulting.
#include "common.cuh"
#include "gemm_host.h"
#include "launch.cuh"
#include "packed_math.cuh"
#include "tcgen05.cuh"

namespace {

using namespace ft;

constexpr int kNV = 4;             // 128-bit pieces of a row per thread

// untiled bulk copy into shared memory (never multicast): both addresses on 16 bytes, bytes a
// multiple of 16
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          sm100::smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(sm100::smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void block_sum2(float& a, float& b, float* scratch /* 64 floats */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  a = warp_sum(a);
  b = warp_sum(b);
  __syncthreads();
  if (lane == 0) { scratch[warp] = a; scratch[32 + warp] = b; }
  __syncthreads();
  float ra = lane < nwarps ? scratch[lane] : 0.f;
  float rb = lane < nwarps ? scratch[32 + lane] : 0.f;
  a = warp_sum(ra);
  b = warp_sum(rb);
}

// Keeps a row piece in its 16-bit form here: left to itself the compiler holds the unpacked floats, twice the
// registers, across the barriers.
__device__ __forceinline__ void stay_packed(uint4& v) { asm volatile("" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)); }

// One CTA per row, H % 8 == 0 and H <= 8 * kNV * blockDim.x.  The CTA has just the threads whose kNV
// pieces cover the row (see launch_norm_fwd): with a fixed 256 threads a 1600-wide row used 200 of
// 1024 piece slots and its two CTA-wide reductions, not memory, set the time (4095 x 1600: 16.9 -> 11.5 us;
// 32768 x 5120 with the residual add: 235 -> 204 us).  w is requested before the reductions and nothing stays
// unpacked across them, so that a row takes 50 to 58 registers a thread: LayerNorm of 32768 x 5120 208 -> 148 us,
// RMSNorm 133 -> 107 us.
// WARP: rows of up to 1024 values, which 32 threads cover, a warp each and up to eight a CTA: as CTAs of one warp they came no faster than
// the machine starts CTAs (us: 2048 x 768 3.6 -> 3.1, 16384 x 768 19.9 -> 12.2, 32768 x 256 35.9 -> 13.6, 4096 x 1024 6.0 -> 5.6).
template <typename T, bool LN, int MAXT, bool WARP>
__global__ void __launch_bounds__(MAXT) norm_fwd_kernel(const T* x, const T* w, const T* b, T* y, float* mean_out,
                                                        float* rstd_out, int64_t rows, int H, float eps, const T* res,
                                                        T* sum_out) {
  __shared__ float red[32];
  wait_previous_kernel();
  const int64_t row = WARP ? (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  const int tid = WARP ? threadIdx.x & 31 : threadIdx.x;
  const int nvec = H / 8, nthr = WARP ? 32 : blockDim.x;
  if (WARP && row >= rows) return;
  auto row_sum = [&](float v) { return WARP ? warp_sum(v) : block_sum(v, red); };
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
  uint4 raw[kNV];
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    const int i = tid + j * nthr;
    raw[j] = i < nvec ? xr[i] : make_uint4(0u, 0u, 0u, 0u);
  }
  if (res != nullptr) {
    // fused residual add: the row that is normalised (and written to sum_out) is x + res,
    // rounded to T first so that the statistics are those of the stored sum
    const uint4* rr = reinterpret_cast<const uint4*>(res + row * H);
    uint4* sr = reinterpret_cast<uint4*>(sum_out + row * H);
    uint4 rraw[kNV];
#pragma unroll
    for (int j = 0; j < kNV; ++j) {
      const int i = tid + j * nthr;
      rraw[j] = i < nvec ? rr[i] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int j = 0; j < kNV; ++j) {
      const int i = tid + j * nthr;
      float a[8], c[8];
      unpack8<T>(raw[j], a);
      unpack8<T>(rraw[j], c);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] += c[k];
      raw[j] = pack8<T>(a);
      if (i < nvec) sr[i] = raw[j];
    }
  }
  // w under the reductions: behind their barriers the compiler has to leave a load where it is written
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4 wraw[kNV];
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    const int i = tid + j * nthr;
    wraw[j] = i < nvec ? wr[i] : make_uint4(0u, 0u, 0u, 0u);
  }
  float mean = 0.f;
  if constexpr (LN) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < kNV; ++j) {
      float v[8];
      unpack8<T>(raw[j], v);                 // pieces past the row hold zeros
#pragma unroll
      for (int k = 0; k < 8; ++k) s += v[k];
    }
    mean = row_sum(s) / (float)H;
#pragma unroll
    for (int j = 0; j < kNV; ++j) stay_packed(raw[j]);
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    if (tid + j * nthr < nvec) {
      float v[8];
      unpack8<T>(raw[j], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += (v[k] - mean) * (v[k] - mean);
    }
  }
  ss = row_sum(ss);
  const float rstd = rsqrtf(ss / (float)H + eps);
  allow_next_kernel();
  if (tid == 0) {
    if (LN) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    stay_packed(raw[j]);
    stay_packed(wraw[j]);
  }
  const uint4* br = reinterpret_cast<const uint4*>(b);
  uint4* yr = reinterpret_cast<uint4*>(y + row * H);
  // every load of b before the first store of y, which it might alias
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    const int i = tid + j * nthr;
    if (i < nvec) {
      float v[8], g[8], o[8];
      unpack8<T>(raw[j], v);
      unpack8<T>(wraw[j], g);
      if constexpr (LN) {
        float bb[8];
        unpack8<T>(br[i], bb);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = (v[k] - mean) * rstd * g[k] + bb[k];
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = v[k] * rstd * g[k];
      }
      raw[j] = pack8<T>(o);
    }
  }
#pragma unroll
  for (int j = 0; j < kNV; ++j) {
    const int i = tid + j * nthr;
    if (i < nvec) yr[i] = raw[j];
  }
}

// Sums N values over the CTA with one pair of barriers; `scratch` holds N * 32 floats.  Returns whether
// `ok` holds in every thread; `between` runs after the first barrier.
template <int N, typename Between>
__device__ __forceinline__ bool block_sum_n(float (&v)[N], float* scratch, bool ok, Between&& between) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int n = 0; n < N; ++n) v[n] = warp_sum(v[n]);
  ok = __syncthreads_and(ok) != 0;
  between();
  if (lane == 0) {
#pragma unroll
    for (int n = 0; n < N; ++n) scratch[n * 32 + warp] = v[n];
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < N; ++n) v[n] = warp_sum(lane < nwarps ? scratch[n * 32 + lane] : 0.f);
  return ok;
}

// Backward of rows of more than 1024 values.  One CTA per SM; a CTA takes R rows per step and each thread NV 128-bit column pieces of
// them (NV * blockDim.x * 8 >= H).  The 2 * R row sums of a step share one CTA-wide reduction.  Every
// CTA leaves one partial row of dw (and db).
//   xh = (x - mean) * rstd, gw = dy * w
//   dx = rstd * (gw - mean(gw) - xh * mean(gw * xh))       (mean(gw) term: LayerNorm only)
// Bound by memory: three or four streams of [rows, H].  x and dy arrive through a ring of `stages`
// steps in shared memory (the R rows of a step are one contiguous piece of each tensor: one bulk copy
// per tensor), so the loads of the next step run under the reductions and stores of this one.  With
// the rows in registers nothing was in flight during those: 356 us for 32768 x 5120 with the residual
// gradient, 253 us with the ring, 201 us being the time of its bytes.  A step's stage is refilled right after the first
// barrier of the next step, which every thread passes only when it has read the stage for the last
// time.  Waits are bounded; one that runs out sets error word 601 and ends the CTA.
constexpr int kBwdRingBytes = 200 * 1024, kBwdMaxStages = 4;

// COPY: dx goes to dx_copy too; as a question in the loop over rows that took 2 to 3 % of every launch.
template <typename T, bool LN, bool COPY, int NV, int R, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) norm_bwd_kernel(const T* x, const T* w, const T* dy,
                                                           const float* mean_in, const float* rstd_in, T* dx,
                                                           float* dw_part, float* db_part, int64_t rows, int H,
                                                           const T* dres, T* dx_copy, int stages, int* err) {
  extern __shared__ uint4 ring[];                    // stages x {x, dy} x R rows
  __shared__ float red[2 * R * 32];
  __shared__ uint64_t full[kBwdMaxStages];
  const int nvec = H / 8;
  const int nthr = blockDim.x;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const int64_t groups = (rows + R - 1) / R;
  const uint32_t row_bytes = (uint32_t)H * 2;
  auto stage_x = [&](int s) { return ring + (int64_t)s * 2 * R * nvec; };
  auto fill = [&](int64_t g, int s) {                // one thread
    const int64_t left = rows - g * R;
    const uint32_t bytes = (uint32_t)(left < R ? left : R) * row_bytes;
    sm100::mbar_expect_tx(&full[s], 2 * bytes);
    bulk_load(stage_x(s), x + g * R * H, bytes, &full[s]);
    bulk_load(stage_x(s) + R * nvec, dy + g * R * H, bytes, &full[s]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) sm100::mbar_init(&full[s], 1);
    sm100::fence_barrier_init();
  }
  __syncthreads();
  wait_previous_kernel();
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      const int64_t g = blockIdx.x + (int64_t)s * gridDim.x;
      if (g < groups) fill(g, s);
    }
  }
  uint4 wraw[NV];
  float dw_acc[NV][8];
  float db_acc[LN ? NV : 1][8];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = threadIdx.x + j * nthr;
    wraw[j] = i < nvec ? wr[i] : zero;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dw_acc[j][k] = 0.f;
      if constexpr (LN) db_acc[j][k] = 0.f;
    }
  }
  const float inv_h = 1.f / (float)H;
  int stage = 0, prev = 0;
  uint32_t phase = 0;
  // mean and rstd of a step's rows are loaded one step ahead: they are four bytes a row, but a read of
  // them at the start of the step is a memory latency in front of everything
  float mean_next[R], rstd_next[R];
  auto load_stats = [&](int64_t g) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t row = g * R + r;
      const bool ok = row < rows;
      mean_next[r] = (LN && ok) ? mean_in[row] : 0.f;
      rstd_next[r] = ok ? rstd_in[row] : 0.f;
    }
  };
  load_stats(blockIdx.x);
  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x) {
    float mean[R], rstd[R];
    uint4 eraw[R][NV];                               // the residual branch's gradient, used at the end
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t row = g * R + r;
      mean[r] = mean_next[r];
      rstd[r] = rstd_next[r];
      if (dres != nullptr) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int i = threadIdx.x + j * nthr;
          eraw[r][j] = row < rows && i < nvec ? reinterpret_cast<const uint4*>(dres + row * H)[i] : zero;
        }
      }
    }
    load_stats(g + gridDim.x);
    bool landed = sm100::mbar_wait(&full[stage], phase);
    const uint4* xs = stage_x(stage);
    const uint4* gs = xs + R * nvec;
    float s[2 * R];
#pragma unroll
    for (int n = 0; n < 2 * R; ++n) s[n] = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (g * R + r < rows) {                        // a row past the end adds nothing anywhere
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int i = threadIdx.x + j * nthr;
          if (i < nvec) {
            float xv[8], gv[8], wv[8];
            unpack8<T>(xs[r * nvec + i], xv);
            unpack8<T>(gs[r * nvec + i], gv);
            unpack8<T>(wraw[j], wv);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float xh = (xv[k] - mean[r]) * rstd[r];
              const float gw = gv[k] * wv[k];
              s[2 * r] += gw;
              s[2 * r + 1] += gw * xh;
              dw_acc[j][k] += gv[k] * xh;
              if constexpr (LN) db_acc[j][k] += gv[k];
            }
          }
        }
      }
    }
    landed = block_sum_n<2 * R>(s, red, landed, [&] {
      // every thread is past the previous step: its stage takes the step `stages` steps after it
      const int64_t next = g + (int64_t)(stages - 1) * gridDim.x;
      if (threadIdx.x == 0 && g != blockIdx.x && next < groups) fill(next, prev);
    });
    if (!landed) {
      if (threadIdx.x == 0) {
        atomicCAS(err, 0, 601);
        // the steps still on their way into this CTA's shared memory
        for (int d = 0; d < stages && g + (int64_t)d * gridDim.x < groups; ++d)
          sm100::mbar_wait(&full[(stage + d) % stages], stage + d < stages ? phase : phase ^ 1u);
      }
      __syncthreads();
      break;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t row = g * R + r;
      if (row < rows) {
        uint4* dr = reinterpret_cast<uint4*>(dx + row * H);
        const float c1 = LN ? s[2 * r] * inv_h : 0.f;
        const float c2 = s[2 * r + 1] * inv_h;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int i = threadIdx.x + j * nthr;
          if (i < nvec) {
            float xv[8], gv[8], wv[8], o[8];
            unpack8<T>(xs[r * nvec + i], xv);
            unpack8<T>(gs[r * nvec + i], gv);
            unpack8<T>(wraw[j], wv);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float xh = (xv[k] - mean[r]) * rstd[r];
              o[k] = rstd[r] * (gv[k] * wv[k] - c1 - xh * c2);
            }
            if (dres != nullptr) {
              // the gradient that reaches the normalised tensor along the residual branch
              float e[8];
              unpack8<T>(eraw[r][j], e);
#pragma unroll
              for (int k = 0; k < 8; ++k) o[k] += e[k];
            }
            const uint4 packed = pack8<T>(o);
            dr[i] = packed;
            if constexpr (COPY) reinterpret_cast<uint4*>(dx_copy + row * H)[i] = packed;
          }
        }
      }
    }
    prev = stage;
    if (++stage == stages) { stage = 0; phase ^= 1; }
  }
  allow_next_kernel();
  float4* ow = reinterpret_cast<float4*>(dw_part + (int64_t)blockIdx.x * H);
  float4* ob = LN ? reinterpret_cast<float4*>(db_part + (int64_t)blockIdx.x * H) : nullptr;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = threadIdx.x + j * nthr;
    if (i < nvec) {
      ow[2 * i] = make_float4(dw_acc[j][0], dw_acc[j][1], dw_acc[j][2], dw_acc[j][3]);
      ow[2 * i + 1] = make_float4(dw_acc[j][4], dw_acc[j][5], dw_acc[j][6], dw_acc[j][7]);
      if constexpr (LN) {
        ob[2 * i] = make_float4(db_acc[j][0], db_acc[j][1], db_acc[j][2], db_acc[j][3]);
        ob[2 * i + 1] = make_float4(db_acc[j][4], db_acc[j][5], db_acc[j][6], db_acc[j][7]);
      }
    }
  }
}

// Backward of rows of up to 1024 values, a warp each: NV 128-bit pieces a lane, no barrier until the rows are done.  In the
// ring above such a row keeps 32 to 128 threads of an SM busy, and they wait for one another twice a step.  LayerNorm with
// the residual gradient, with the sum of the partial rows, us: 256 x 256 5.4 -> 4.3, 1024 x 768 8.0 -> 6.6, 2048 x 768 11.6 -> 8.0,
// 16384 x 768 61 -> 25 (15 being the time of its bytes), 32768 x 256 33 -> 15.  Groups of threads with a ring each: 8.2, 28 and 20.
// As many warps as keep a lane's sums and its row in registers.
__host__ __device__ constexpr int norm_warps(int nv, bool ln) { return nv == 1 || (ln && (nv == 2 || nv == 4)) ? 8 : 12; }

template <typename T, bool LN, bool COPY, int NV>
__global__ void __launch_bounds__(32 * norm_warps(NV, LN), 4 / NV)
norm_bwd_warp_kernel(const T* x, const T* w, const T* dy, const float* mean_in, const float* rstd_in, T* dx, float* dw_part,
                     float* db_part, int64_t rows, int H, const T* dres, T* dx_copy) {
  constexpr int WARPS = norm_warps(NV, LN);
  __shared__ float4 sums[WARPS][NV * 64];
  wait_previous_kernel();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nvec = H / 8;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const float inv_h = 1.f / (float)H;
  uint4 wraw[NV];
  float dw_acc[NV][8], db_acc[LN ? NV : 1][8];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = lane + j * 32;
    wraw[j] = i < nvec ? reinterpret_cast<const uint4*>(w)[i] : zero;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dw_acc[j][k] = 0.f;
      if constexpr (LN) db_acc[j][k] = 0.f;
    }
  }
  for (int64_t row = (int64_t)warp * gridDim.x + blockIdx.x; row < rows; row += (int64_t)WARPS * gridDim.x) {
    const uint4 *xr = reinterpret_cast<const uint4*>(x + row * H), *gr = reinterpret_cast<const uint4*>(dy + row * H);
    uint4 xraw[NV], graw[NV], eraw[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {                   // pieces past the row hold zeros and add nothing
      const int i = lane + j * 32;
      xraw[j] = i < nvec ? xr[i] : zero;
      graw[j] = i < nvec ? gr[i] : zero;
    }
    if (dres != nullptr) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const int i = lane + j * 32;
        eraw[j] = i < nvec ? reinterpret_cast<const uint4*>(dres + row * H)[i] : zero;
      }
    }
    const float mean = LN ? mean_in[row] : 0.f, rstd = rstd_in[row];
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float xv[8], gv[8], wv[8];
      unpack8<T>(xraw[j], xv);
      unpack8<T>(graw[j], gv);
      unpack8<T>(wraw[j], wv);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float xh = (xv[k] - mean) * rstd, gw = gv[k] * wv[k];
        c1 += gw;
        c2 += gw * xh;
        dw_acc[j][k] += gv[k] * xh;
        if constexpr (LN) db_acc[j][k] += gv[k];
      }
    }
    c1 = LN ? warp_sum(c1) * inv_h : 0.f;
    c2 = warp_sum(c2) * inv_h;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * 32;
      if (i < nvec) {
        float xv[8], gv[8], wv[8], o[8];
        unpack8<T>(xraw[j], xv);
        unpack8<T>(graw[j], gv);
        unpack8<T>(wraw[j], wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = rstd * (gv[k] * wv[k] - c1 - (xv[k] - mean) * rstd * c2);
        if (dres != nullptr) {
          float e[8];
          unpack8<T>(eraw[j], e);
#pragma unroll
          for (int k = 0; k < 8; ++k) o[k] += e[k];
        }
        const uint4 packed = pack8<T>(o);
        reinterpret_cast<uint4*>(dx + row * H)[i] = packed;
        if constexpr (COPY) reinterpret_cast<uint4*>(dx_copy + row * H)[i] = packed;
      }
    }
  }
  allow_next_kernel();
  // the sums of the warps that had rows, one vector after the other
  const int64_t mine = (rows - blockIdx.x + gridDim.x - 1) / gridDim.x;
  const int busy = mine < WARPS ? (int)mine : WARPS;
  auto leave = [&](const float (&acc)[NV][8], float* out) {
    if (warp < busy) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        float4* at = &sums[warp][2 * (lane + j * 32)];
        at[0] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        at[1] = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * nvec; i += 32 * WARPS) {
      float4 t = sums[0][i];
#pragma unroll 4
      for (int v = 1; v < busy; ++v) {
        const float4 a = sums[v][i];
        t.x += a.x; t.y += a.y; t.z += a.z; t.w += a.w;
      }
      reinterpret_cast<float4*>(out + (int64_t)blockIdx.x * H)[i] = t;
    }
  };
  leave(dw_acc, dw_part);
  if constexpr (LN) {
    __syncthreads();
    leave(db_acc, db_part);
  }
}

// out[c] (+)= sum_p part[p][c], for some (part, out) pairs: the partial rows a backward kernel left, one per CTA.  Bound by latency, the partials sit in L2: with one thread per
// column walking all the rows (up to 148) a 1600-wide reduction took 8 us; with 32 columns x 32 row
// lanes per CTA every thread has at most five independent loads (both sums of a LayerNorm: 16.1 -> 3.2 us).
constexpr int kPartCols = 32, kPartRows = 32;

// The sums of one launch: those of a LayerNorm's two vectors, or all that a block's backward leaves for its end (each launch of its own
// was 3 us on the device and as much on the host).  Sum i has the columns' CTAs from first[i] on.
constexpr int kPartSums = 6;
struct PartSums {
  const float* part[kPartSums];
  void* out[kPartSums];
  int parts[kPartSums], N[kPartSums], first[kPartSums], add[kPartSums];
  int n;
};

template <typename T>
__global__ void __launch_bounds__(kPartCols * kPartRows)
parts_reduce_kernel(const __grid_constant__ PartSums sums) {
  __shared__ float red[kPartRows][kPartCols + 1];
  wait_previous_kernel();
  int i = 0;
  while (i + 1 < sums.n && (int)blockIdx.x >= sums.first[i + 1]) ++i;
  const float* part = sums.part[i];
  T* out = static_cast<T*>(sums.out[i]);
  const int parts = sums.parts[i], N = sums.N[i];
  const int col = threadIdx.x % kPartCols, lane = threadIdx.x / kPartCols;
  const int c = ((int)blockIdx.x - sums.first[i]) * kPartCols + col;
  float s = 0.f;
  if (c < N) {
#pragma unroll 5
    for (int p = lane; p < parts; p += kPartRows) s += part[(int64_t)p * N + c];
  }
  red[lane][col] = s;
  allow_next_kernel();
  __syncthreads();
  if (lane == 0 && c < N) {
    float t = sums.add[i] ? to_float(out[c]) : 0.f;
#pragma unroll
    for (int r = 0; r < kPartRows; ++r) t += red[r][col];
    out[c] = from_float<T>(t);
  }
}

template <typename T>
void launch_part_sums(PartSums& sums, cudaStream_t s) {
  int blocks = 0;
  int64_t bytes = 0;
  for (int i = 0; i < sums.n; ++i) {
    sums.first[i] = blocks;
    blocks += (sums.N[i] + kPartCols - 1) / kPartCols;
    bytes += (int64_t)sums.parts[i] * sums.N[i] * 4;
  }
  launch_overlapped(parts_reduce_kernel<T>, blocks, kPartCols * kPartRows, 0, s, 1, overlap_bytes(bytes), sums);
}

// bit i of `accumulate`: out i is added to
template <typename T>
void launch_parts_reduce(const float* part0, void* out0, const float* part1, void* out1, int parts, int N,
                         int accumulate, cudaStream_t s) {
  PartSums sums{{part0, part1}, {out0, out1}, {parts, parts}, {N, N}, {}, {accumulate & 1, accumulate >> 1 & 1}, part1 ? 2 : 1};
  launch_part_sums<T>(sums, s);
}

// ------------------------------------------------------------ bias + activation
// The tanh GELU, 0.5 u (1 + tanh z) with z = sqrt(2 / pi) (u + 0.044715 u^3), is u s(2 z) with the logistic function
// s(x) = 1 / (1 + e^-x), and its derivative s + u s (1 - s) 2 z'.  That is one exponential and one quotient with nothing
// that cancels (tanh written out as 1 - 2 / (1 + e^2z) does for negative u), and the polynomials go two values at a time.
constexpr float kGeluK = 0.7978845608028654f;    // sqrt(2 / pi)
constexpr float kGeluC = 0.044715f;
constexpr float kLog2E = 1.4426950408889634f;

// e^(-2 z) of two values
__device__ __forceinline__ void gelu_exp2(uint64_t u, uint64_t uu, float& e0, float& e1) {
  constexpr float a = -2.f * kGeluK * kLog2E, b = a * kGeluC;
  float x0, x1;
  pm::unpack2(pm::mul2(u, pm::fma2(uu, pm::pack2(b, b), pm::pack2(a, a))), x0, x1);
  e0 = pm::ex2(x0);
  e1 = pm::ex2(x1);
}

__device__ __forceinline__ void gelu_tanh2(float u0, float u1, float& y0, float& y1) {
  const uint64_t u = pm::pack2(u0, u1);
  float e0, e1;
  gelu_exp2(u, pm::mul2(u, u), e0, e1);
  y0 = __fdividef(u0, 1.f + e0);                   // 0 where the denominator overflows
  y1 = __fdividef(u1, 1.f + e1);
}

// The derivative is 0 or 1 to the last bit from |u| = 16 on; u is held there, because u 2 z' overflows from 1e13 on
// where s or 1 - s is 0.  NaN stays NaN.
constexpr float kGeluFlat = 16.f;

__device__ __forceinline__ float gelu_hold(float u) {
  asm("min.NaN.f32 %0, %0, %1;\n\tmax.NaN.f32 %0, %0, %2;" : "+f"(u) : "f"(kGeluFlat), "f"(-kGeluFlat));
  return u;
}

__device__ __forceinline__ void gelu_tanh_grad2(float u0, float u1, float& d0, float& d1) {
  constexpr float a = 2.f * kGeluK, b = 3.f * a * kGeluC;
  u0 = gelu_hold(u0);
  u1 = gelu_hold(u1);
  const uint64_t u = pm::pack2(u0, u1), uu = pm::mul2(u, u), one = pm::pack2(1.f, 1.f);
  float e0, e1;
  gelu_exp2(u, uu, e0, e1);
  const uint64_t s = pm::pack2(__fdividef(1.f, 1.f + e0), __fdividef(1.f, 1.f + e1));
  const uint64_t slope = pm::mul2(u, pm::fma2(uu, pm::pack2(b, b), pm::pack2(a, a)));      // u 2 z'
  const uint64_t rest = pm::fma2(s, pm::pack2(-1.f, -1.f), one);
  pm::unpack2(pm::mul2(s, pm::fma2(rest, slope, one)), d0, d1);
}

// x, y: [rows, N] with row stride N; y may alias x.  ACT 0: identity, 1: tanh GELU.
// CTA = 2^lg columns of eight x 256 / 2^lg row lanes of ROWS rows each, all loaded before the first is used; grid
// (columns, row blocks).  A flat loop over vectors took a 64-bit remainder for the column of each and had one load in
// flight: 3000 x 6400 29 us where its bytes take 12.  See BiasShape for lg and ROWS.
constexpr int kBiasRows = 4;

template <typename T, int ACT, int ROWS>
__global__ void __launch_bounds__(256) bias_act_fwd_kernel(const T* x, const T* bias, T* y, int64_t rows, int N, int lg) {
  wait_previous_kernel();
  const int vec = N / 8, lanes = 256 >> lg;
  const int c = ((int)blockIdx.x << lg) + (threadIdx.x & ((1 << lg) - 1));
  const int64_t r0 = (int64_t)blockIdx.y * (lanes * ROWS) + (threadIdx.x >> lg);
  if (c < vec) {
    uint4 raw[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
      if (r0 + lanes * i < rows) raw[i] = reinterpret_cast<const uint4*>(x)[(r0 + lanes * i) * vec + c];
    float bb[8];
    unpack8<T>(reinterpret_cast<const uint4*>(bias)[c], bb);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      if (r0 + lanes * i < rows) {
        float o[8];
        unpack8<T>(raw[i], o);
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          o[k] += bb[k];
          o[k + 1] += bb[k + 1];
          if constexpr (ACT == 1) gelu_tanh2(o[k], o[k + 1], o[k], o[k + 1]);
        }
        reinterpret_cast<uint4*>(y)[(r0 + lanes * i) * vec + c] = pack8<T>(o);
      }
    }
  }
  allow_next_kernel();
}

// CTA = 32 column groups (8 columns each) x 8 row lanes; grid (ceil(N / 256), parts).
// dx = dy * act'(x + bias) (not written when dx == nullptr, i.e. identity);
// db_part[blockIdx.y][c] = sum over this CTA's rows of dx[:, c].
template <typename T, int ACT>
__global__ void __launch_bounds__(256) bias_act_bwd_kernel(const T* dy, const T* x, const T* bias, T* dx,
                                                           float* db_part, int64_t rows, int N) {
  __shared__ float red[8][257];
  wait_previous_kernel();
  const int vec = N / 8;
  const int cg = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cg;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  if (c < vec) {
    float bb[8];
    if (ACT == 1) unpack8<T>(reinterpret_cast<const uint4*>(bias)[c], bb);
    // kBiasRows rows a step, all loaded before the first is used
    const int64_t step = (int64_t)gridDim.y * 8;
    for (int64_t r0 = (int64_t)blockIdx.y * 8 + rl; r0 < rows; r0 += kBiasRows * step) {
      uint4 graw[kBiasRows], xraw[kBiasRows];
#pragma unroll
      for (int i = 0; i < kBiasRows; ++i) {
        const int64_t r = r0 + i * step;
        if (r < rows) {
          graw[i] = reinterpret_cast<const uint4*>(dy)[r * vec + c];
          if (ACT == 1) xraw[i] = reinterpret_cast<const uint4*>(x)[r * vec + c];
        }
      }
#pragma unroll
      for (int i = 0; i < kBiasRows; ++i) {
        const int64_t r = r0 + i * step;
        if (r < rows) {
          float g[8];
          unpack8<T>(graw[i], g);
          if constexpr (ACT == 1) {
            float v[8], o[8];
            unpack8<T>(xraw[i], v);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
              float d0, d1;
              gelu_tanh_grad2(v[k] + bb[k], v[k + 1] + bb[k + 1], d0, d1);
              o[k] = g[k] * d0;
              o[k + 1] = g[k + 1] * d1;
              acc[k] += o[k];
              acc[k + 1] += o[k + 1];
            }
            reinterpret_cast<uint4*>(dx)[r * vec + c] = pack8<T>(o);
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += g[k];
          }
        }
      }
    }
  }
  allow_next_kernel();
#pragma unroll
  for (int k = 0; k < 8; ++k) red[rl][cg * 8 + k] = acc[k];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < N) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) s += red[r][threadIdx.x];
    db_part[(int64_t)blockIdx.y * N + col] = s;
  }
}

// ------------------------------------------------------------ embedding, backward
// grad[token] += the sum of the rows of dy [n, H] whose token it is, in fp32 with one rounding and in a fixed order (the same bits every
// time): one CTA a row of dy, and a token's CTAs divide its columns, so that a token that comes often, as padding does, has as many CTAs as
// it can use.  A look at n tokens for each of n rows is little beside what the general way does for it, a zeroed gradient of the whole table,
// a scatter and an addition of the two.  Rows that name no token of the table are left out.
// us with the launch, 768 columns of 50304 tokens, random tokens / three quarters of them one / all of them one: 1024 rows 12 / 11 / 10 (the
// general way 112 / 130 / 138), 4096 rows 35 / 28 / 23 (240 / 231 / 234); 4096 rows of 8192 columns, 128256 tokens, 84 / 53 / 33 (2117 / 1869 /
// 1789).  One CTA for all rows of a token took 573 and 2 280 for 1024 and 4096 rows of one.
constexpr int kEmbedThreads = 256, kEmbedMost = 4096;      // rows of dy
constexpr int kEmbedRows = 8;                        // under way a thread
constexpr int kEmbedSlice = 4;                       // vectors of a token's row that a CTA takes at least

template <typename T>
__global__ void __launch_bounds__(kEmbedThreads, 4) embedding_add_kernel(const int64_t* tokens, const T* dy, T* grad, int n, int H, int64_t V) {
  __shared__ uint16_t rows[kEmbedMost];
  __shared__ int2 found[kEmbedThreads / 32];
  __shared__ float4 sums[2][kEmbedThreads];
  wait_previous_kernel();
  const int row = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nvec = H / 8;
  const int64_t token = tokens[row];
  if (token < 0 || token >= V) return;
  // this warp's share of the rows of the token, and of those before this one
  int2 mine = make_int2(0, 0);
#pragma unroll 4
  for (int base = 0; base < n; base += kEmbedThreads) {
    const int j = base + tid;
    const bool same = j < n && tokens[j] == token;
    mine.x += __popc(__ballot_sync(0xffffffffu, same));
    mine.y += __popc(__ballot_sync(0xffffffffu, same && j < row));
  }
  if (lane == 0) found[warp] = mine;
  __syncthreads();
  int count = 0, before = 0, at = 0;
#pragma unroll
  for (int w = 0; w < kEmbedThreads / 32; ++w) {
    at += w < warp ? found[w].x : 0;
    count += found[w].x;
    before += found[w].y;
  }
  const int slices = min(count, (nvec + kEmbedSlice - 1) / kEmbedSlice), share = (nvec + slices - 1) / slices;
  const int begin = before * share, end = min(nvec, begin + share);
  if (begin >= end) return;
  if (count == 1) {
    if (tid == 0) rows[0] = (uint16_t)row;
  } else {
#pragma unroll 4
    for (int base = 0; base < n; base += kEmbedThreads) {
      const int j = base + tid;
      const bool same = j < n && tokens[j] == token;
      const unsigned votes = __ballot_sync(0xffffffffu, same);
      if (same) rows[at + __popc(votes & ((1u << lane) - 1))] = (uint16_t)j;
      at += __popc(votes);
    }
  }
  __syncthreads();
  // threads of a row, and rows at a time
  int width = 1;
  while (width < share && width < kEmbedThreads) width *= 2;
  const int group = tid / width, groups = kEmbedThreads / width;
  for (int first = begin; first < end; first += width) {
    const int i = first + tid % width;
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    for (int m = group; i < end && m < count; m += groups * kEmbedRows) {
      uint4 raw[kEmbedRows];
#pragma unroll
      for (int u = 0; u < kEmbedRows; ++u) {
        const int r = m + u * groups;
        raw[u] = r < count ? reinterpret_cast<const uint4*>(dy + (int64_t)rows[r] * H)[i] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < kEmbedRows; ++u) {
        float v[8];
        unpack8<T>(raw[u], v);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += v[k];
      }
    }
    if (first + width >= end) allow_next_kernel();
    if (groups > 1 && count > 1) {
      sums[0][tid] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      sums[1][tid] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      __syncthreads();
      for (int g = 1; group == 0 && g < groups && g < count; ++g) {
        const float4 a = sums[0][g * width + tid], b = sums[1][g * width + tid];
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
        acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
      }
      __syncthreads();
    }
    if (group == 0 && i < end) {
      uint4* out = reinterpret_cast<uint4*>(grad + token * H) + i;
      float v[8];
      unpack8<T>(*out, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += acc[k];
      *out = pack8<T>(v);
    }
  }
}

#define FT_DISPATCH_16(dt, T, ...)                            \
  if (dt == kBF16) { using T = __nv_bfloat16; __VA_ARGS__; }  \
  else if (dt == kF16) { using T = __half; __VA_ARGS__; }     \
  else return -1;

inline int round_up32(int v) { return (v + 31) / 32 * 32; }

template <typename T, bool LN>
void launch_norm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                     int64_t rows, int H, float eps, const void* res, void* sum_out, cudaStream_t s) {
  const int nvec = H / 8;
  const int threads = round_up32((nvec + kNV - 1) / kNV);
  // rows of one warp: four CTAs of them an SM first, then up to eight rows a CTA, two where a row takes all the pieces of its warp
  const int most = H > 768 ? 2 : 8, warps = threads > 32 ? 0 : rows < 148 * 8 ? 1 : rows < 148 * 4 * most ? (int)(rows / (148 * 4)) : most;
#define FT_NORM_FWD(MAXT, WARP, GRID, THREADS)                                                         \
  launch_overlapped(norm_fwd_kernel<T, LN, MAXT, WARP>, (unsigned)(GRID), THREADS, 0, s, 1, overlap_bytes(rows * H * 4),   \
                    (const T*)x, (const T*)w,                                                          \
                    (const T*)b, (T*)y, mean, rstd, rows, H, eps, (const T*)res, (T*)sum_out)
  if (warps > 0) FT_NORM_FWD(256, true, (rows + warps - 1) / warps, 32 * warps);
  else if (threads <= 256) FT_NORM_FWD(256, false, rows, threads);
  else FT_NORM_FWD(1024, false, rows, threads);
#undef FT_NORM_FWD
}

// Shape of the ring's launch: pieces per thread, rows per step, threads.  A step costs two barriers and a wait
// whatever its rows hold, so rows of up to 2048 values go eight at a time where there are enough of them.  With four
// the ring was slower than rows in registers had been: 4095 x 1600 18.1 -> 20.3 us, 16.2 so.
struct BwdShape { int nv, r, threads; };
inline BwdShape norm_bwd_shape(int64_t rows, int H) {
  const int nvec = H / 8;
  if (nvec <= 256 && rows >= 148 * 16) return {1, 8, round_up32(nvec)};
  if (nvec <= 640) return {1, 4, round_up32(nvec)};
  if (nvec <= 1024) return {2, 2, round_up32((nvec + 1) / 2)};
  return {4, 1, round_up32((nvec + 3) / 4)};
}

template <typename T, bool LN, bool COPY>
void launch_norm_bwd(const void* x, const void* w, const void* dy, const float* mean, const float* rstd,
                     void* dx, float* dw_part, float* db_part, int64_t rows, int H, int parts,
                     const void* dres, void* dx_copy, cudaStream_t s) {
  if (H <= 1024) {
#define FT_NORM_BWD_WARP(NV)                                                                                      \
  launch_overlapped(norm_bwd_warp_kernel<T, LN, COPY, NV>, parts, 32 * norm_warps(NV, LN), 0, s, 1, overlap_bytes(rows * H * 6), \
                    (const T*)x, (const T*)w, (const T*)dy, mean, rstd, (T*)dx, dw_part, db_part, rows, H,        \
                    (const T*)dres, (T*)dx_copy)
    if (H <= 256) FT_NORM_BWD_WARP(1);
    else if (H <= 512) FT_NORM_BWD_WARP(2);
    else if (H <= 768) FT_NORM_BWD_WARP(3);
    else FT_NORM_BWD_WARP(4);
#undef FT_NORM_BWD_WARP
    return;
  }
  const BwdShape sh = norm_bwd_shape(rows, H);
  const int stage_bytes = 2 * sh.r * H * 2;
  int stages = kBwdRingBytes / stage_bytes;
  if (stages > kBwdMaxStages) stages = kBwdMaxStages;
  int dev = 0;
  cudaGetDevice(&dev);
  int* err = gemm::error_word(dev);
#define FT_NORM_BWD(NV, R, MAXT)                                                                      \
  {                                                                                                   \
    auto kern = norm_bwd_kernel<T, LN, COPY, NV, R, MAXT>;                                            \
    static DynamicSmem smem;                                                                          \
    smem.grant(kern, kBwdRingBytes);                                                                  \
    launch_overlapped(kern, parts, sh.threads, stages * stage_bytes, s, 1, overlap_bytes(rows * H * 6),  \
                      (const T*)x, (const T*)w,                                                       \
                      (const T*)dy, mean, rstd, (T*)dx, dw_part, db_part, rows, H, (const T*)dres,    \
                      (T*)dx_copy, stages, err);                                                                   \
  }
  if (sh.r == 8) FT_NORM_BWD(1, 8, 256)
  else if (sh.nv == 1 && sh.threads <= 512) FT_NORM_BWD(1, 4, 512)
  else if (sh.nv == 1) FT_NORM_BWD(1, 4, 640)
  else if (sh.nv == 2) FT_NORM_BWD(2, 2, 512)
  else FT_NORM_BWD(4, 1, 512)
#undef FT_NORM_BWD
}

}  // namespace

extern "C" {

// Largest hidden size of ft_norm_fwd / ft_norm_bwd_into.
int ft_norm_max_hidden(int backward) { return backward ? 8 * 4 * 512 : 8 * kNV * 1024; }

// Number of partial rows ft_norm_bwd_into writes into dw_part / db_part: one per CTA.  The ring: one CTA per SM, or one a step.
// A warp a row: rows / 4 up to one CTA an SM.  Where a row is narrow the sum of the partial rows takes as long as the rows, so up to 1280
// rows of up to 512 values have 64 CTAs at most, and two CTAs an SM (four of up to 256 values) come where there are enough rows.  LayerNorm
// with the residual gradient and the sum, us with 64 / 148 / 296 / 592 CTAs: 1000 x 256 4.8 / 5.5 / 6.2 / 8.0, 2300 x 256 6.6 / 6.2 / 6.7 / 8.5,
// 12000 x 256 - / 12.0 / 10.4 / 11.1, 65536 x 256 - / 61 / 41 / 31, 4096 x 512 - / 7.9 / 8.5, 6000 x 512 - / 10.2 / 9.4; without the sum, which a
// block's backward forms at its end, 1000 x 768 4.5 / 3.3 / 4.7.  With as many CTAs as the ring had, rows / 4 up to 592, 1820 x 256 took
// 7.6 where the ring took 6.7.
int ft_norm_bwd_parts(int64_t rows, int H) {
  if (H > 0 && H % 8 == 0 && H <= 1024) {
    const int64_t some = rows < 1 ? 1 : (rows + 3) / 4;
    const int most = H > 512 ? 148 : rows <= 1280 ? 64 : rows < 5000 ? 148 : H > 256 || rows < 20480 ? 296 : 592;
    return (int)(some < most ? some : most);
  }
  const BwdShape sh = H % 8 == 0 && H > 0 ? norm_bwd_shape(rows, H) : BwdShape{1, 1, 128};
  const int64_t groups = (rows + sh.r - 1) / sh.r;
  return (int)(groups < 1 ? 1 : groups < 148 ? groups : 148);
}

// layernorm != 0: y = (x - mean) * rstd * w + b, mean and rstd saved per row.
// layernorm == 0: y = x * rstd * w (b, mean unused; may be null).
// With `res` (and `sum_out`) the row that is normalised is x + res, which is also written to
// sum_out in the tensors' dtype: the residual add before a norm costs no pass of its own.
int ft_add_norm_fwd(const void* x, const void* res, void* sum_out, const void* w, const void* b, void* y,
                    float* mean, float* rstd, int64_t rows, int H, float eps, int layernorm, int dt,
                    cudaStream_t s) {
  if (rows <= 0) return 0;
  if (H % 8 || H > ft_norm_max_hidden(0)) return -2;
  if (!aligned16(x) || !aligned16(w) || !aligned16(y) || (layernorm && !aligned16(b))) return -2;
  if ((res == nullptr) != (sum_out == nullptr)) return -2;
  if (res && (!aligned16(res) || !aligned16(sum_out))) return -2;
  if (rows > 0x7fffffffLL) return -2;
  FT_DISPATCH_16(dt, T, {
    if (layernorm) launch_norm_fwd<T, true>(x, w, b, y, mean, rstd, rows, H, eps, res, sum_out, s);
    else launch_norm_fwd<T, false>(x, w, nullptr, y, nullptr, rstd, rows, H, eps, res, sum_out, s);
  });
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_norm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                int64_t rows, int H, float eps, int layernorm, int dt, cudaStream_t s) {
  return ft_add_norm_fwd(x, nullptr, nullptr, w, b, y, mean, rstd, rows, H, eps, layernorm, dt, s);
}

// dw_part (and db_part for LayerNorm): ft_norm_bwd_parts(rows, H) * H floats of scratch.
// dw / db receive the column sums in the parameters' dtype `dt`, added to what they hold where bit 0 / bit 1
// of `accumulate` is set.
// Without dw (nullptr) the partial rows are left in dw_part and db_part, for ft_sum_parts.
// With `dres` ([rows, H], same dtype) dx = dres + (gradient through the norm): the sum of the two
// gradient branches that meet at the norm's input is formed here (dx and dres are distinct buffers).
// With `dx_copy` dx is written there too: two leaves whose sum was normalised need a buffer each, and copying one to
// the other reads again what this kernel holds in registers (32768 x 5120, forward + backward: 556 -> 474 us).
int ft_norm_bwd_into(const void* x, const void* w, const void* dy, const void* dres, const float* mean,
                     const float* rstd, void* dx, void* dx_copy, void* dw, void* db, float* dw_part, float* db_part,
                     int64_t rows, int H, int layernorm, int accumulate, int dt, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (H % 8 || H > ft_norm_max_hidden(1)) return -2;
  if (!aligned16(x) || !aligned16(w) || !aligned16(dy) || !aligned16(dx) || !aligned16(dw_part) ||
      (layernorm && !aligned16(db_part)) || (dres && !aligned16(dres)) || (dx_copy && !aligned16(dx_copy)))
    return -2;
  const int parts = ft_norm_bwd_parts(rows, H);
  FT_DISPATCH_16(dt, T, {
    auto* launch = layernorm ? (dx_copy ? launch_norm_bwd<T, true, true> : launch_norm_bwd<T, true, false>)
                             : (dx_copy ? launch_norm_bwd<T, false, true> : launch_norm_bwd<T, false, false>);
    launch(x, w, dy, layernorm ? mean : nullptr, rstd, dx, dw_part, layernorm ? db_part : nullptr, rows, H, parts, dres,
           dx_copy, s);
    if (dw != nullptr) launch_parts_reduce<T>(dw_part, dw, layernorm ? db_part : nullptr, db, parts, H, accumulate, s);
  });
  FT_LAUNCHED(dw != nullptr ? 2 : 1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int N, int act, int dt, cudaStream_t s);

// Launch shape of the forward.  lg: as many column lanes as the rows have vectors, at most 32: with 32 for every
// width most of a warp had nothing to do for rows below 256 values (GELU, 65536 x 8: 10.3 us, now 1.7; 2^20 x 64: 139, now 40).
// ROWS: four once one each fills the device, because a thread's rows follow one another (87 x 568: 2.27 us, now 1.67).
constexpr int64_t kBiasFew = 148 * 1024;                 // vectors up to which a thread takes one row
struct BiasShape { int lg, rows; int64_t block_rows; };

static BiasShape bias_shape(int64_t rows, int N) {
  const int vec = N / 8;
  int lg = 0;
  while (lg < 5 && (1 << lg) < vec) ++lg;
  const int n = rows * vec <= kBiasFew ? 1 : kBiasRows;
  return {lg, n, (int64_t)(256 >> lg) * n};
}

// More rows than a grid's second dimension holds (at least 2 million): one launch after another.
static int bias_act_in_parts(const void* x, const void* bias, void* y, int64_t rows, int N, int act, int dt,
                             cudaStream_t s) {
  const int64_t most = 65535LL * bias_shape(rows, N).block_rows;
  for (int64_t r = 0; r < rows; r += most) {
    const int64_t bytes = r * N * 2;
    const int rc = ft_bias_act_fwd(static_cast<const char*>(x) + bytes, bias, static_cast<char*>(y) + bytes,
                                   rows - r < most ? rows - r : most, N, act, dt, s);
    if (rc) return rc;
  }
  return 0;
}

// y = act(x + bias) over [rows, N]; y may be x.  act 0: identity, 1: tanh GELU.
int ft_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int N, int act, int dt,
                    cudaStream_t s) {
  if (rows <= 0) return 0;
  if (N % 8 || (act != 0 && act != 1)) return -2;
  if (!aligned16(x) || !aligned16(bias) || !aligned16(y)) return -2;
  const BiasShape sh = bias_shape(rows, N);
  const int64_t blocks = (rows + sh.block_rows - 1) / sh.block_rows;
  if (blocks > 65535) return bias_act_in_parts(x, bias, y, rows, N, act, dt, s);
  const dim3 grid((N / 8 + (1 << sh.lg) - 1) >> sh.lg, (unsigned)blocks);
  FT_DISPATCH_16(dt, T, {
    auto* kern = sh.rows == 1 ? (act == 1 ? bias_act_fwd_kernel<T, 1, 1> : bias_act_fwd_kernel<T, 0, 1>)
                              : (act == 1 ? bias_act_fwd_kernel<T, 1, kBiasRows> : bias_act_fwd_kernel<T, 0, kBiasRows>);
    launch_overlapped(kern, grid, 256, 0, s, 1, overlap_bytes(rows * N * 4), (const T*)x, (const T*)bias, (T*)y, rows, N, sh.lg);
  });
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// Number of partial rows ft_bias_act_bwd writes for a [rows, N] problem.
int ft_bias_act_bwd_parts(int64_t rows, int N) {
  const int gx = (N + 255) / 256;
  int64_t parts = (148 * 8 + gx - 1) / gx;
  const int64_t by_rows = (rows + 7) / 8;
  if (parts > by_rows) parts = by_rows;
  if (parts > 64) parts = 64;
  if (parts < 1) parts = 1;
  return (int)parts;
}

// dx = dy * act'(x + bias) (act 1; for act 0 dx is dy itself and x, dx are unused),
// dbias (+)= column sums of dx (nullptr: the partial rows are left for ft_sum_parts).  db_part: ft_bias_act_bwd_parts(rows, N) * N floats.
int ft_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx, void* dbias,
                    float* db_part, int64_t rows, int N, int act, int accumulate, int dt,
                    cudaStream_t s) {
  if (rows <= 0) return 0;
  if (N % 8 || (act != 0 && act != 1)) return -2;
  if (!aligned16(dy)) return -2;
  if (act == 1 && (!aligned16(x) || !aligned16(bias) || !aligned16(dx))) return -2;
  const int parts = ft_bias_act_bwd_parts(rows, N);
  const dim3 grid((N + 255) / 256, parts);
  FT_DISPATCH_16(dt, T, {
    launch_overlapped(act == 1 ? bias_act_bwd_kernel<T, 1> : bias_act_bwd_kernel<T, 0>, grid, 256, 0, s, 1,
                      overlap_bytes(rows * N * (act ? 6 : 2)),
                      (const T*)dy, (const T*)x, (const T*)bias, (T*)dx, db_part, rows, N);
    if (dbias != nullptr) launch_parts_reduce<T>(db_part, dbias, nullptr, nullptr, parts, N, accumulate != 0, s);
  });
  FT_LAUNCHED(dbias != nullptr ? 2 : 1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// out[i][c] (+)= the sum of the `parts[i]` rows of part[i], N[i] columns wide, for n of up to six: the partial rows that
// ft_norm_bwd_into and ft_bias_act_bwd were told to leave, in one launch.
int ft_sum_parts(int n, const float* const* part, void* const* out, const int* parts, const int* N, const int* add, int dt,
                 cudaStream_t s) {
  if (n < 0 || n > kPartSums) return -2;
  if (n == 0) return 0;
  PartSums sums{};
  sums.n = n;
  for (int i = 0; i < n; ++i) {
    sums.part[i] = part[i];
    sums.out[i] = out[i];
    sums.parts[i] = parts[i];
    sums.N[i] = N[i];
    sums.add[i] = add[i];
  }
  FT_DISPATCH_16(dt, T, launch_part_sums<T>(sums, s));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// grad [V, H] += dy [n, H] by token, where the tokens are few (`n` up to 4096) and a row has up to 8192 values; -4 for what it does not take.
int ft_embedding_add(const int64_t* tokens, const void* dy, void* grad, int64_t n, int H, int64_t V, int dt, cudaStream_t s) {
  if (n <= 0) return 0;
  if (n > kEmbedMost || H <= 0 || H % 8 || H > 8192 || !aligned16(dy) || !aligned16(grad)) return -4;
  FT_DISPATCH_16(dt, T, launch_overlapped(embedding_add_kernel<T>, (unsigned)n, kEmbedThreads, 0, s, 1, overlap_bytes(n * H * 6),
                                          tokens, (const T*)dy, (T*)grad, (int)n, H, V));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

}  // extern "C"
