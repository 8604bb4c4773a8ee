// Host stand-ins for the C entry points that csrc/torch calls (bf16 only), so that what the autograd
// nodes do with layouts, buffers and autograd can be tested without a GPU.  Products, rope and the bias
// add are the real functions; attention hands q, k and v through, which shows where they are read and
// written.  Load with RTLD_GLOBAL before libft_torch.so.
#include <c10/cuda/CUDAStream.h>

#include <cstring>
#include <vector>

#pragma GCC visibility push(default)
namespace c10::cuda {
CUDAStream getCurrentCUDAStream(DeviceIndex) {
  return CUDAStream(CUDAStream::UNCHECKED, c10::Stream(c10::Stream::UNSAFE, c10::Device(c10::DeviceType::CUDA, 0), 0));
}
cudaStream_t CUDAStream::stream() const { return nullptr; }
}  // namespace c10::cuda

namespace {
float get(const void* p, int64_t i) {
  const uint32_t bits = (uint32_t)((const uint16_t*)p)[i] << 16;
  float f;
  memcpy(&f, &bits, 4);
  return f;
}
void put(void* p, int64_t i, float f) {
  uint32_t bits;
  memcpy(&bits, &f, 4);
  ((uint16_t*)p)[i] = (uint16_t)((bits + 0x7fff + ((bits >> 16) & 1)) >> 16);
}
void copy_rows(const void* src, int64_t src_stride, void* dst, int64_t dst_stride, int64_t rows, int64_t width) {
  for (int64_t r = 0; r < rows; ++r)
    memcpy((uint16_t*)dst + r * dst_stride, (const uint16_t*)src + r * src_stride, width * 2);
}
int rope_in_place = 0, rope_calls = 0, backward_launches = 0, sum_launches = 0, embedding_launches = 0;

// column sums of a [rows, N], times `scale`: left in `part`, or added to or stored in `out`
void column_sums(const void* a, int64_t rows, int N, float scale, void* out, bool add, float* part) {
  std::vector<float> s(N, 0.f);
  for (int64_t i = 0; i < rows * N; ++i) s[i % N] += scale * get(a, i);
  for (int n = 0; n < N; ++n) {
    if (out == nullptr) part[n] = s[n];
    else put(out, n, s[n] + (add ? get(out, n) : 0.f));
  }
}
}  // namespace

extern "C" {
int stub_rope_in_place() { return rope_in_place; }   // how many calls had x = y
int stub_rope_calls() { return rope_calls; }
int stub_backward_launches() { return backward_launches; }
int stub_sum_launches() { return sum_launches; }
int stub_embedding_launches() { return embedding_launches; }

int ft_gemm_bias(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc, int,
                 int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K, int, void*) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;             // as the real one: C is left alone
  for (int64_t m = 0; m < M; ++m)
    for (int64_t n = 0; n < N; ++n) {
      float s = bias ? get(bias, n) : 0.f;
      for (int64_t k = 0; k < K; ++k)
        s += get(A, a_mn ? k * lda + m : m * lda + k) * get(B, b_mn ? k * ldb + n : n * ldb + k);
      if (R) s += get(R, m * ldr + n);
      else if (accumulate) s += get(C, m * ldc + n);
      put(C, m * ldc + n, s);
    }
  return 0;
}

// asks for a workspace where k is a multiple of three
int64_t ft_gemm_ws_bytes(int, int, int K, int) { return K % 3 ? 0 : 64; }
int ft_gemm_ws(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc, int dt,
               int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K, int ab, void* ws,
               int64_t bytes, void* s) {
  if (bytes < 0 && K % 3 == 0) return -5;
  if (bytes > 0 && (K % 3 || bytes < 64 || !ws)) return -9;
  return ft_gemm_bias(A, a_mn, lda, B, b_mn, ldb, C, ldc, dt, accumulate, R, ldr, bias, M, N, K, ab, s);
}

// sums on the way for an even number of rows
int ft_gemm_dw_db(const void* dy, int64_t ldy, const void* x, int64_t ldx, void* dw, int64_t ldw, int add_dw, void* db,
                  int add_db, int T, int N, int K, int dt, void* s) {
  if (T <= 0 || T % 2) return -4;
  for (int n = 0; n < N; ++n) {
    float sum = add_db ? get(db, n) : 0.f;
    for (int64_t t = 0; t < T; ++t) sum += get(dy, t * ldy + n);
    put(db, n, sum);
  }
  return ft_gemm_bias(dy, 1, ldy, x, 1, ldx, dw, ldw, dt, add_dw, nullptr, 0, nullptr, N, K, T, dt, s);
}

// one launch for both products where the number of rows is a multiple of four
int ft_gemm_backward(const void* dy, int64_t ldy, const void* w, int64_t ldw, const void* x, int64_t ldx, void* dx, int64_t ldx2,
                     void* dw, int64_t ld_dw, int add_dw, void* db, int add_db, int t, int n, int k, int dt, void* s) {
  if (t <= 0 || t % 4) return -4;
  backward_launches++;
  ft_gemm_bias(dy, 0, ldy, w, 1, ldw, dx, ldx2, dt, 0, nullptr, 0, nullptr, t, k, n, dt, s);
  if (db) return ft_gemm_dw_db(dy, ldy, x, ldx, dw, ld_dw, add_dw, db, add_db, t, n, k, dt, s);
  return ft_gemm_bias(dy, 1, ldy, x, 1, ldx, dw, ld_dw, dt, add_dw, nullptr, 0, nullptr, n, k, t, dt, s);
}

int ft_rope(const void* x, int64_t xs, void* y, int64_t ys, const float* cos_t, const float* sin_t, int64_t tokens,
            int heads, int D, int seq_len, float sign, int, void*) {
  rope_calls++;
  rope_in_place += x == y;
  const int half = D / 2;
  for (int64_t t = 0; t < tokens; ++t)
    for (int h = 0; h < heads; ++h)
      for (int i = 0; i < half; ++i) {
        const int64_t tab = t % seq_len * half + i, a = t * xs + h * D + i, o = t * ys + h * D + i;
        const float u = get(x, a), v = get(x, a + half), c = cos_t[tab], s = sign * sin_t[tab];
        put(y, o, u * c - v * s);
        put(y, o + half, v * c + u * s);
      }
  return 0;
}

// act 1 doubles: not a GELU, but what is read and written where
int ft_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int N, int act, int, void*) {
  if (rows <= 0) return 0;
  for (int64_t i = 0; i < rows * N; ++i) put(y, i, (act ? 2.f : 1.f) * (get(x, i) + get(bias, i % N)));
  return 0;
}
int ft_bias_act_bwd_parts(int64_t, int) { return 1; }
int ft_bias_act_bwd(const void* dy, const void*, const void*, void* dx, void* dbias, float* part, int64_t rows, int N, int act,
                    int accumulate, int, void*) {
  if (rows <= 0) return 0;
  for (int64_t i = 0; act && i < rows * N; ++i) put(dx, i, 2.f * get(dy, i));
  column_sums(act ? dx : dy, rows, N, 1.f, dbias, accumulate, part);
  return 0;
}

int ft_attn_fwd(const void* q, int64_t qs, const void*, int64_t, const void*, int64_t, void* o, float*, int B, int S,
                int Hq, int, int D, float, int, void*) {
  copy_rows(q, qs, o, (int64_t)Hq * D, (int64_t)B * S, (int64_t)Hq * D);
  return 0;
}
int ft_attn_bwd_parts(int, int, int, int, int) { return 1; }
int ft_attn_bwd_split(const void* q, int64_t qs, const void* k, int64_t ks, const void* v, int64_t vs, const void*,
                      const void*, int64_t, const float*, float*, float*, float*, int, void* dq, int64_t dqs, void* dk,
                      int64_t dks, void* dv, int64_t dvs, int B, int S, int Hq, int Hkv, int D, float, int, void*,
                      long long*, int, int) {
  copy_rows(q, qs, dq, dqs, (int64_t)B * S, (int64_t)Hq * D);
  copy_rows(k, ks, dk, dks, (int64_t)B * S, (int64_t)Hkv * D);
  copy_rows(v, vs, dv, dvs, (int64_t)B * S, (int64_t)Hkv * D);
  return 0;
}

// these tests give them nothing to do
int ft_gemm_swiglu(const void*, int64_t, const void*, int64_t, void*, int64_t, void*, int64_t, int M, int, int, int,
                   void*) {
  return M <= 0 ? 0 : -1;
}
int ft_swiglu_fwd(const void*, void*, int64_t rows, int, int, void*) { return rows <= 0 ? 0 : -1; }
int ft_swiglu_bwd(const void*, const void*, void*, int64_t rows, int, int, void*) { return rows <= 0 ? 0 : -1; }
// y = sum_out = x (+ res): not a norm, but what is read and written where
int ft_add_norm_fwd(const void* x, const void* res, void* sum_out, const void*, const void*, void* y, float*, float*,
                    int64_t rows, int H, float, int, int, void*) {
  for (int64_t i = 0; i < rows * H; ++i) {
    put(y, i, get(x, i) + (res ? get(res, i) : 0.f));
    if (sum_out) put(sum_out, i, get(y, i));
  }
  return 0;
}
int ft_norm_bwd_parts(int64_t, int) { return 1; }
// dx = dy (+ dres), dw = column sums of dy, db = twice that: not a norm, but what is written where
int ft_norm_bwd_into(const void*, const void*, const void* dy, const void* dres, const float*, const float*, void* dx,
                     void* dx_copy, void* dw, void* db, float* dw_part, float* db_part, int64_t rows, int H, int layernorm,
                     int accumulate, int, void*) {
  if (rows <= 0) return 0;
  for (int64_t i = 0; i < rows * H; ++i) {
    put(dx, i, get(dy, i) + (dres ? get(dres, i) : 0.f));
    if (dx_copy) put(dx_copy, i, get(dx, i));
  }
  column_sums(dy, rows, H, 1.f, dw, accumulate & 1, dw_part);
  if (layernorm) column_sums(dy, rows, H, 2.f, db, accumulate >> 1 & 1, db_part);
  return 0;
}

// Every sum of a launch reads what it adds to before any of them writes, as its CTAs may.
int ft_sum_parts(int n, const float* const* part, void* const* out, const int* parts, const int* N, const int* add, int, void*) {
  sum_launches++;
  std::vector<std::vector<float>> sums(n);
  for (int i = 0; i < n; ++i)
    for (int c = 0; c < N[i]; ++c) {
      float s = add[i] ? get(out[i], c) : 0.f;
      for (int p = 0; p < parts[i]; ++p) s += part[i][(int64_t)p * N[i] + c];
      sums[i].push_back(s);
    }
  for (int i = 0; i < n; ++i)
    for (int c = 0; c < N[i]; ++c) put(out[i], c, sums[i][c]);
  return 0;
}

// takes an even number of rows
int ft_embedding_add(const int64_t* tokens, const void* dy, void* grad, int64_t n, int H, int64_t V, int, void*) {
  if (n % 2) return -4;
  embedding_launches++;
  for (int64_t i = 0; i < n; ++i)
    for (int h = 0; tokens[i] >= 0 && tokens[i] < V && h < H; ++h)
      put(grad, tokens[i] * H + h, get(grad, tokens[i] * H + h) + get(dy, i * H + h));
  return 0;
}
}
