// Bandwidth-bound model ops of the Llama block, bf16/fp16/fp32 I/O with fp32
// math: RMSNorm (fwd, bwd), rotary embedding (fwd = bwd with the sign of sin
// flipped; strided input or output so it reads / writes slices of the fused QKV
// tensor directly), SwiGLU (fwd, bwd) and the softmax cross-entropy row kernels
// used by the chunked head (row log-sum-exp + loss; in-place dlogits).
//
// The reference has no model code: these replace the ATen kernels a user model
// would call.  One 128-bit access per thread per step; rows are processed by
// one CTA each so every reduction stays on chip.
#include <type_traits>

#include "common.cuh"
#include "launch.cuh"

namespace {

using namespace ft;

// ----------------------------------------------------------------- RMSNorm
// y = x * rsqrt(mean(x^2) + eps) * w ; inv_rms saved per row.  H % 8 == 0.
template <typename T>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const T* __restrict__ x,
                                                          const T* __restrict__ w, T* __restrict__ y,
                                                          float* __restrict__ inv_rms, int H, float eps) {
  __shared__ float red[32];
  const int64_t row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + row * H);
  const int nvec = H / 8;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float v[8];
    unpack8<T>(xr[i], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0) inv_rms[row] = inv;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float v[8], g[8], o[8];
    unpack8<T>(xr[i], v);
    unpack8<T>(wr[i], g);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = v[k] * inv * g[k];
    yr[i] = pack8<T>(o);
  }
}

// dx = inv * (g*w - x * inv^2 * mean(g*w*x)); partial dw per CTA (rows strided by grid).
template <typename T>
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(const T* __restrict__ x,
                                                          const T* __restrict__ w,
                                                          const T* __restrict__ dy,
                                                          const float* __restrict__ inv_rms,
                                                          T* __restrict__ dx, float* __restrict__ dw_part,
                                                          int64_t rows, int H) {
  __shared__ float red[32];
  const int nvec = H / 8;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  constexpr int kMaxVec = 8;   // per-thread column groups kept in registers: H <= 8 * 8 * 256
  float dw_acc[kMaxVec][8];
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j)
#pragma unroll
    for (int k = 0; k < 8; ++k) dw_acc[j][k] = 0.f;

  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + row * H);
    uint4* dr = reinterpret_cast<uint4*>(dx + row * H);
    const float inv = inv_rms[row];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < kMaxVec; ++j) {
      int i = threadIdx.x + j * blockDim.x;
      if (i < nvec) {
        float xv[8], gv[8], wv[8];
        unpack8<T>(xr[i], xv);
        unpack8<T>(gr[i], gv);
        unpack8<T>(wr[i], wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          dot += gv[k] * wv[k] * xv[k];
          dw_acc[j][k] += gv[k] * xv[k] * inv;
        }
      }
    }
    dot = block_sum(dot, red);
    const float coef = dot * inv * inv / (float)H;
#pragma unroll
    for (int j = 0; j < kMaxVec; ++j) {
      int i = threadIdx.x + j * blockDim.x;
      if (i < nvec) {
        float xv[8], gv[8], wv[8], o[8];
        unpack8<T>(xr[i], xv);
        unpack8<T>(gr[i], gv);
        unpack8<T>(wr[i], wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = inv * (gv[k] * wv[k] - xv[k] * coef);
        dr[i] = pack8<T>(o);
      }
    }
  }
  float* out = dw_part + (int64_t)blockIdx.x * H;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    int i = threadIdx.x + j * blockDim.x;
    if (i < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) out[i * 8 + k] = dw_acc[j][k];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) rmsnorm_dw_reduce_kernel(const float* __restrict__ part,
                                                                T* __restrict__ dw, int parts, int H) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= H) return;
  float s = 0.f;
  for (int p = 0; p < parts; ++p) s += part[(int64_t)p * H + c];
  dw[c] = from_float<T>(s);
}

// -------------------------------------------------------------------- RoPE
// x viewed as [tokens, heads, D] with token strides in elements; rotate-half
// pairs (i, i + D/2); position = token % seq_len.  sin_sign = -1 gives the
// transpose rotation (backward).  One thread per (token, 8 columns of the first half, range of
// `heads_per` heads): it loads its 8 cosines and sines once and walks its heads, four at a time, so
// the tables are read once per token and range instead of once per head and eight 16-byte loads are
// in flight per thread; what is left after the fours is read at once too (100000 tokens of 3 heads: 37.7 us head by
// head, 31.2 us so).  blockIdx.y is the range; see ft_rope for how many there are.
template <typename T>
__device__ __forceinline__ void rope_rotate8(const uint4& xa, const uint4& xb, const float (&c)[8],
                                             const float (&s)[8], uint4& ya, uint4& yb) {
  float a[8], b[8], oa[8], ob[8];
  unpack8<T>(xa, a);
  unpack8<T>(xb, b);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    oa[k] = a[k] * c[k] - b[k] * s[k];
    ob[k] = b[k] * c[k] + a[k] * s[k];
  }
  ya = pack8<T>(oa);
  yb = pack8<T>(ob);
}

template <typename T>
__global__ void __launch_bounds__(256) rope_kernel(const T* x, int64_t x_tok_stride, T* y,
                                                   int64_t y_tok_stride, const float* cos_t,
                                                   const float* sin_t, int64_t tokens, int heads, int heads_per,
                                                   int D, int seq_len, float sin_sign) {
  wait_previous_kernel();
  const int half = D / 2, vec = half / 8;
  const int h_begin = blockIdx.y * heads_per, h_end = min(heads, h_begin + heads_per);
  const int64_t total = tokens * vec;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)(idx % vec);
    const int64_t tok = idx / vec;
    const int pos = (int)(tok % seq_len);
    float c[8], s[8];
    const float4* cp = reinterpret_cast<const float4*>(cos_t + (int64_t)pos * half + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + (int64_t)pos * half + v * 8);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    s[0] = s0.x; s[1] = s0.y; s[2] = s0.z; s[3] = s0.w; s[4] = s1.x; s[5] = s1.y; s[6] = s1.z; s[7] = s1.w;
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] *= sin_sign;
    const T* xp = x + tok * x_tok_stride + v * 8;
    T* yp = y + tok * y_tok_stride + v * 8;
    auto turn = [&](int h, auto count) {               // all loads before any store: x may be y
      constexpr int N = decltype(count)::value;
      uint4 xa[N], xb[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        xa[u] = *reinterpret_cast<const uint4*>(xp + (int64_t)(h + u) * D);
        xb[u] = *reinterpret_cast<const uint4*>(xp + (int64_t)(h + u) * D + half);
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        uint4 ya, yb;
        rope_rotate8<T>(xa[u], xb[u], c, s, ya, yb);
        *reinterpret_cast<uint4*>(yp + (int64_t)(h + u) * D) = ya;
        *reinterpret_cast<uint4*>(yp + (int64_t)(h + u) * D + half) = yb;
      }
    };
    int h = h_begin;
    for (; h + 4 <= h_end; h += 4) turn(h, std::integral_constant<int, 4>());
    const int rest = h_end - h;
    if (rest == 3) turn(h, std::integral_constant<int, 3>());
    else if (rest == 2) turn(h, std::integral_constant<int, 2>());
    else if (rest == 1) turn(h, std::integral_constant<int, 1>());
  }
  allow_next_kernel();
}

// ------------------------------------------------------------------ SwiGLU
// in: [rows, 2F] = [gate | up]; out: [rows, F].
template <typename T>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const T* gu, T* out, int64_t rows, int F) {
  wait_previous_kernel();
  const int vec = F / 8;
  const int64_t total = rows * vec;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / vec;
    const int c = (int)(idx % vec) * 8;
    float g[8], u[8], o[8];
    unpack8<T>(*reinterpret_cast<const uint4*>(gu + r * 2 * F + c), g);
    unpack8<T>(*reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = __fdividef(g[k], 1.f + __expf(-g[k])) * u[k];
    *reinterpret_cast<uint4*>(out + r * F + c) = pack8<T>(o);
  }
  allow_next_kernel();
}

template <typename T>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const T* gu, const T* dout, T* dgu, int64_t rows,
                                                         int F) {
  wait_previous_kernel();
  const int vec = F / 8;
  const int64_t total = rows * vec, step = (int64_t)gridDim.x * blockDim.x;
  int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  // the next piece is read before this one's results are stored, which it might alias
  uint4 graw, uraw, draw;
  auto load = [&](int64_t i) {
    if (i >= total) return;
    const T* p = gu + i / vec * 2 * F + i % vec * 8;
    graw = *reinterpret_cast<const uint4*>(p);
    uraw = *reinterpret_cast<const uint4*>(p + F);
    draw = reinterpret_cast<const uint4*>(dout)[i];
  };
  load(idx);
  for (; idx < total; idx += step) {
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8<T>(graw, g);
    unpack8<T>(uraw, u);
    unpack8<T>(draw, d);
    load(idx + step);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float sig = __fdividef(1.f, 1.f + __expf(-g[k]));   // approximate reciprocal: the result is rounded to 16 bits
      float silu = g[k] * sig;
      dg[k] = d[k] * u[k] * sig * (1.f + g[k] * (1.f - sig));
      du[k] = d[k] * silu;
    }
    T* q = dgu + idx / vec * 2 * F + idx % vec * 8;
    *reinterpret_cast<uint4*>(q) = pack8<T>(dg);
    *reinterpret_cast<uint4*>(q + F) = pack8<T>(du);
  }
  allow_next_kernel();
}

// ----------------------------------------------------- softmax cross-entropy
// One CTA per row of logits [rows, V] (row stride ld).  Forward: lse[row] and the
// row's loss (0 for ignored labels) accumulated into *loss_sum.  Backward (in
// place): logits <- (softmax - onehot) * (*grad_scale_ptr) * inv_count, rows with
// an ignored label become 0.
//
// Both kernels are bound by the bytes of the logits, so the forward reads each row once: every thread
// keeps a running maximum and the sum relative to it, four 16-byte pieces in flight, and the CTA
// merges the pairs at the end.  (4095 x 32000: 139 us with the maximum first and the sum in a second
// sweep, 66 us so, 40 us being the time of the bytes; backward 106 -> 83 us, 80 us for its bytes.)
constexpr int kXentAhead = 4;

struct MaxSum {
  float m = -INFINITY, s = 0.f;
  // n values; a thread that has met only -inf sums against 0, so that a masked piece adds 0 and a NaN
  // still reaches the sum
  template <int N>
  __device__ __forceinline__ void add(const float (&v)[N]) {
    float vm = v[0];
#pragma unroll
    for (int k = 1; k < N; ++k) vm = fmaxf(vm, v[k]);
    if (vm > m) {
      s *= __expf(m - vm);                             // first piece: 0 * e^-inf
      m = vm;
    }
    const float ref = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int k = 0; k < N; ++k) s += __expf(v[k] - ref);
  }
};

template <typename T>
__device__ __forceinline__ void row_max_sum(const T* row, int V, float* red, float& mx, float& sum) {
  const int nvec = V / 8;
  const uint4* rv = reinterpret_cast<const uint4*>(row);
  MaxSum a;
  int i = threadIdx.x;
  for (; i + (kXentAhead - 1) * (int)blockDim.x < nvec; i += kXentAhead * blockDim.x) {
    uint4 raw[kXentAhead];
#pragma unroll
    for (int u = 0; u < kXentAhead; ++u) raw[u] = rv[i + u * blockDim.x];
#pragma unroll
    for (int u = 0; u < kXentAhead; ++u) {
      float v[8];
      unpack8<T>(raw[u], v);
      a.add(v);
    }
  }
  for (; i < nvec; i += blockDim.x) {
    float v[8];
    unpack8<T>(rv[i], v);
    a.add(v);
  }
  for (i = nvec * 8 + threadIdx.x; i < V; i += blockDim.x) {
    const float v[1] = {to_float(row[i])};
    a.add(v);
  }
  mx = block_max(a.m, red);
  // a row of nothing but -inf has no softmax: NaN, as -inf - -inf gives
  sum = block_sum(a.m == mx ? a.s : a.s * __expf(a.m - mx), red);
  if (mx == -INFINITY) sum = NAN;
}

template <typename T>
__global__ void __launch_bounds__(512) xent_fwd_kernel(const T* logits, int64_t ld,
                                                       const int64_t* labels, int V,
                                                       int64_t ignore_index, float* lse,
                                                       float* loss_sum) {
  __shared__ float red[32];
  wait_previous_kernel();
  const int64_t r = blockIdx.x;
  const T* row = logits + r * ld;
  float mx, sum;
  row_max_sum<T>(row, V, red, mx, sum);
  allow_next_kernel();
  if (threadIdx.x == 0) {
    float l = mx + logf(sum);
    lse[r] = l;
    int64_t lab = labels[r];
    if (lab != ignore_index && lab >= 0 && lab < V) atomicAdd(loss_sum, l - to_float(row[lab]));
  }
}

// Threads of a row: four pieces each and at least 128.  With 512 whatever the row, 1024 columns kept three of four
// threads idle and the SM's slots full of them: 4096 x 1024 11.0 us, 5.6 us so; 1000 x 8192 7.9 -> 5.5 us.
inline int xent_bwd_threads(int V) {
  const int t = (V / 8 / kXentAhead + 31) / 32 * 32;
  return t < 128 ? 128 : t > 512 ? 512 : t;
}

template <typename T>
__global__ void __launch_bounds__(512) xent_bwd_kernel(T* logits, int64_t ld,
                                                       const int64_t* labels, int V,
                                                       int64_t ignore_index,
                                                       const float* lse,
                                                       const float* grad_out,
                                                       float inv_count) {
  wait_previous_kernel();
  const int64_t r = blockIdx.x;
  T* row = logits + r * ld;
  const int64_t lab64 = labels[r];
  const bool valid = lab64 != ignore_index && lab64 >= 0 && lab64 < V;
  const int lab = valid ? (int)lab64 : -1;
  const float scale = valid ? (*grad_out) * inv_count : 0.f;
  const float l = lse[r];
  const int nvec = V / 8;
  uint4* rv = reinterpret_cast<uint4*>(row);
  auto piece = [&](int i, const uint4& raw) {
    float v[8], o[8];
    unpack8<T>(raw, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = (__expf(v[k] - l) - (i * 8 + k == lab ? 1.f : 0.f)) * scale;
    rv[i] = pack8<T>(o);
  };
  int i = threadIdx.x;
  for (; i + (kXentAhead - 1) * (int)blockDim.x < nvec; i += kXentAhead * blockDim.x) {
    uint4 raw[kXentAhead];
#pragma unroll
    for (int u = 0; u < kXentAhead; ++u) raw[u] = rv[i + u * blockDim.x];
#pragma unroll
    for (int u = 0; u < kXentAhead; ++u) piece(i + u * blockDim.x, raw[u]);
  }
  for (; i < nvec; i += blockDim.x) piece(i, rv[i]);
  allow_next_kernel();
  for (i = nvec * 8 + threadIdx.x; i < V; i += blockDim.x)
    row[i] = from_float<T>((__expf(to_float(row[i]) - l) - (i == lab ? 1.f : 0.f)) * scale);
}

__global__ void count_valid_kernel(const int64_t* __restrict__ labels, int64_t n, int64_t ignore_index,
                                   int V, int* __restrict__ count) {
  int local = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t lab = labels[i];
    local += (lab != ignore_index && lab >= 0 && lab < V) ? 1 : 0;
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, local);
}

#define FT_DISPATCH_16(dt, T, ...)                            \
  if (dt == kBF16) { using T = __nv_bfloat16; __VA_ARGS__; }  \
  else if (dt == kF16) { using T = __half; __VA_ARGS__; }     \
  else return -1;

}  // namespace

extern "C" {

int ft_rmsnorm_fwd(const void* x, const void* w, void* y, float* inv_rms, int64_t rows, int H,
                   float eps, int dt, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (H % 8) return -2;
  FT_DISPATCH_16(dt, T, (rmsnorm_fwd_kernel<T><<<(unsigned)rows, 256, 0, s>>>(
                            (const T*)x, (const T*)w, (T*)y, inv_rms, H, eps)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// dw_part: scratch of parts * H floats; parts returned by ft_rmsnorm_bwd_parts().
int ft_rmsnorm_bwd_parts() { return 148 * 2; }

int ft_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* inv_rms, void* dx,
                   void* dw, float* dw_part, int64_t rows, int H, int dt, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (H % 8 || H > 8 * 8 * 256) return -2;
  int parts = ft_rmsnorm_bwd_parts();
  if (parts > rows) parts = (int)rows;
  FT_DISPATCH_16(dt, T, {
    rmsnorm_bwd_kernel<T><<<parts, 256, 0, s>>>((const T*)x, (const T*)w, (const T*)dy, inv_rms, (T*)dx,
                                                 dw_part, rows, H);
    rmsnorm_dw_reduce_kernel<T><<<(H + 255) / 256, 256, 0, s>>>(dw_part, (T*)dw, parts, H);
  });
  FT_LAUNCHED(1);
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_rope(const void* x, int64_t x_tok_stride, void* y, int64_t y_tok_stride, const float* cos_t,
            const float* sin_t, int64_t tokens, int heads, int D, int seq_len, float sin_sign, int dt,
            cudaStream_t s) {
  if (tokens <= 0) return 0;
  if (D % 16 || x_tok_stride % 8 || y_tok_stride % 8) return -2;
  if (!aligned16(x) || !aligned16(y) || !aligned16(cos_t) || !aligned16(sin_t)) return -2;
  if (heads <= 0) return 0;
  const int grid = grid_for(tokens * (D / 16), 256);
  // Enough CTAs to keep the memory system busy (eight per SM): with one thread for all the heads of a
  // token, 4096 tokens are 128 CTAs on 148 SMs (50 us for 64 heads of 128 in place, 134 MB; 24 us with
  // eight ranges).  Ranges are multiples of the four heads a thread has in flight.
  int ranges = (148 * 8 + grid - 1) / grid;
  if (ranges > (heads + 3) / 4) ranges = (heads + 3) / 4;
  const int heads_per = ((heads + ranges - 1) / ranges + 3) / 4 * 4;
  ranges = (heads + heads_per - 1) / heads_per;
  FT_DISPATCH_16(dt, T, (launch_overlapped(rope_kernel<T>, dim3(grid, ranges), 256, 0, s, 1, overlap_bytes(tokens * heads * D * 4),
                            (const T*)x, x_tok_stride, (T*)y, y_tok_stride, cos_t, sin_t, tokens, heads,
                            heads_per, D, seq_len, sin_sign)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_swiglu_fwd(const void* gu, void* out, int64_t rows, int F, int dt, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (F % 8 || !aligned16(gu) || !aligned16(out)) return -2;
  FT_DISPATCH_16(dt, T, (launch_overlapped(swiglu_fwd_kernel<T>, grid_for(rows * (F / 8), 256), 256, 0, s, 1, overlap_bytes(rows * F * 6),
                            (const T*)gu, (T*)out, rows, F)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_swiglu_bwd(const void* gu, const void* dout, void* dgu, int64_t rows, int F, int dt,
                  cudaStream_t s) {
  if (rows <= 0) return 0;
  if (F % 8 || !aligned16(gu) || !aligned16(dout) || !aligned16(dgu)) return -2;
  FT_DISPATCH_16(dt, T, (launch_overlapped(swiglu_bwd_kernel<T>, grid_for(rows * (F / 8), 256), 256, 0, s, 1, overlap_bytes(rows * F * 10),
                            (const T*)gu, (const T*)dout, (T*)dgu, rows, F)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_xent_fwd(const void* logits, int64_t ld, const int64_t* labels, int64_t rows, int V,
                int64_t ignore_index, float* lse, float* loss_sum, int dt, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (ld % 8) return -2;
  FT_DISPATCH_16(dt, T, (launch_overlapped(xent_fwd_kernel<T>, (unsigned)rows, 512, 0, s, 1, overlap_bytes(rows * V * 2),
                            (const T*)logits, ld, labels, V, ignore_index, lse, loss_sum)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_xent_bwd(void* logits, int64_t ld, const int64_t* labels, int64_t rows, int V,
                int64_t ignore_index, const float* lse, const float* grad_out, float inv_count, int dt,
                cudaStream_t s) {
  if (rows <= 0) return 0;
  if (ld % 8) return -2;
  FT_DISPATCH_16(dt, T, (launch_overlapped(xent_bwd_kernel<T>, (unsigned)rows, xent_bwd_threads(V), 0, s, 1, overlap_bytes(rows * V * 4),
                            (T*)logits, ld, labels, V, ignore_index, lse, grad_out, inv_count)));
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

int ft_count_valid(const int64_t* labels, int64_t n, int64_t ignore_index, int V, int* count,
                   cudaStream_t s) {
  if (n <= 0) return 0;
  count_valid_kernel<<<grid_for(n, 256, 148), 256, 0, s>>>(labels, n, ignore_index, V, count);
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

}  // extern "C"
