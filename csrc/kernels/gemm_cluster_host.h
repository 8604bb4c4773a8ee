// Launches of the cluster GEMM (gemm_cluster.cuh).
#pragma once
#include "gemm_cluster.cuh"
#include "gemm_host.h"

namespace ft {
namespace gemm {
namespace {                                          // what a launch keeps belongs to the library that includes this

struct ClusterProduct {
  const void *A, *B;
  void* C;
  const void *R, *bias;    // R: the matrix that is added (C for +=), nullptr: none
  int64_t lda, ldb, ldc, ldr;
  int a_mn, b_mn, M, N, K, dtype;
  void* row_sum;
  int row_sum_add;
};

// Shared memory of a CTA at most: with the kilobyte that the system takes of each, two fit an SM.
constexpr int C_SMEM_BYTES = 115712;

// Stages of the ring.  Three or more, which hold the tile (and, where it is divided, the other pair's sums).
inline int cluster_stages(int tn, bool b_mn) {
  const int n = (C_SMEM_BYTES - C_RING_OFFSET - 1024) / cluster_stage_bytes(tn, b_mn);
  return n < C_MAX_STAGES ? n : C_MAX_STAGES;
}

template <typename T, bool A_MN, bool B_MN, bool ACC, int TN>
int launch_cluster_one(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tr,
                       const ClusterArgs& args, cudaStream_t s) {
  auto kern = gemm_cluster_kernel<T, A_MN, B_MN, ACC, TN>;
  static DynamicSmem smem;
  smem.grant(kern, C_SMEM_BYTES);
  cudaError_t e = launch_overlapped(kern, args.mt * args.nt * 2 * args.splits, C_THREADS,
                                    C_RING_OFFSET + args.stages * cluster_stage_bytes(TN, B_MN) + 1024, s, 2 * args.splits,
                                    overlap_product(args.M, args.N, args.K), ta, tb, tc, tr, args);
  return e == cudaSuccess ? 0 : (int)e;
}

template <typename T, bool A_MN, bool B_MN, bool ACC>
int launch_cluster_tile(int tile_n, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tr,
                        const ClusterArgs& args, cudaStream_t s) {
  switch (tile_n) {
    case 64: return launch_cluster_one<T, A_MN, B_MN, ACC, 64>(ta, tb, tc, tr, args, s);
    case 128: return launch_cluster_one<T, A_MN, B_MN, ACC, 128>(ta, tb, tc, tr, args, s);
    case 192: return launch_cluster_one<T, A_MN, B_MN, ACC, 192>(ta, tb, tc, tr, args, s);
    default: return launch_cluster_one<T, A_MN, B_MN, ACC, 256>(ta, tb, tc, tr, args, s);
  }
}

inline ClusterArgs cluster_args(int M, int N, int K, bool b_mn, int tile_n, int splits, int group_m, const void* bias, void* row_sum,
                                int row_sum_add, int* err) {
  const int kt = (K + BK - 1) / BK, stages = cluster_stages(tile_n, b_mn);
  return {M, N, K, splits, stages, kt % stages, (M + P_BM - 1) / P_BM, (N + tile_n - 1) / tile_n, kt, group_m, bias, row_sum, row_sum_add, err};
}

template <typename T>
int launch_cluster(const ClusterProduct& p, int tile_n, int splits, int group_m, cudaStream_t s) {
  int dev = 0;
  cudaGetDevice(&dev);
  CUtensorMap ta, tb, tc, tr;
  int rc = p.a_mn ? make_tmap(&ta, p.A, p.M, p.K, p.lda, 64, BK, p.dtype) : make_tmap(&ta, p.A, p.K, p.M, p.lda, BK, BM, p.dtype);
  if (rc == 0)
    rc = p.b_mn ? make_tmap(&tb, p.B, p.N, p.K, p.ldb, 64, BK, p.dtype)
                : make_tmap(&tb, p.B, p.K, p.N, p.ldb, BK, tile_n / 2, p.dtype);
  if (rc == 0) rc = make_tmap(&tc, p.C, p.N, p.M, p.ldc, 64, BM, p.dtype);
  if (rc == 0) rc = p.R != nullptr ? make_tmap(&tr, p.R, p.N, p.M, p.ldr, 64, BM, p.dtype) : (tr = tc, 0);
  if (rc) return rc;
  const ClusterArgs args = cluster_args(p.M, p.N, p.K, p.b_mn, tile_n, splits, group_m, p.bias, p.row_sum, p.row_sum_add, error_word(dev));
#define FT_CLUSTER(A_MN, B_MN)                                                                                   \
  return p.R != nullptr ? launch_cluster_tile<T, A_MN, B_MN, true>(tile_n, ta, tb, tc, tr, args, s)       \
                        : launch_cluster_tile<T, A_MN, B_MN, false>(tile_n, ta, tb, tc, tr, args, s)
  if (!p.a_mn && !p.b_mn) FT_CLUSTER(false, false);
  if (!p.a_mn) FT_CLUSTER(false, true);
  if (p.b_mn) FT_CLUSTER(true, true);
#undef FT_CLUSTER
  return -4;
}

// The products of a projection's backward pass: dy [t, n], w [n, k], x [t, k], dx [t, k], dw [n, k].
struct BackwardProducts {
  const void *dy, *w, *x;
  void *dx, *dw, *row_sum;
  int64_t ld_dy, ld_w, ld_x, ld_dx, ld_dw;
  int t, n, k, add_dw, row_sum_add, dtype;
};

template <typename T, bool ACC, int TN>
int launch_backward_one(const CUtensorMap (&m)[6], const ClusterArgs& dx, const ClusterArgs& dw, cudaStream_t s) {
  auto kern = gemm_cluster_backward_kernel<T, ACC, TN>;
  static DynamicSmem smem;
  smem.grant(kern, C_SMEM_BYTES);
  const int blocks_dx = dx.mt * dx.nt * 2 * dx.splits, blocks_dw = dw.mt * dw.nt * 2 * dw.splits;
  const int dw_first = dw.kt > dx.kt;
  cudaError_t e = launch_overlapped(kern, blocks_dx + blocks_dw, C_THREADS, C_RING_OFFSET + dx.stages * cluster_stage_bytes(TN, true) + 1024,
                                    s, 2 * dx.splits, overlap_product(dx.M, dx.N, 2LL * dx.K), m[0], m[1], m[2], m[3], m[4], m[5], dx, dw,
                                    dw_first ? blocks_dw : blocks_dx, dw_first);
  return e == cudaSuccess ? 0 : (int)e;
}

template <typename T, bool ACC>
int launch_backward_tile(int tile_n, const CUtensorMap (&m)[6], const ClusterArgs& dx, const ClusterArgs& dw, cudaStream_t s) {
  switch (tile_n) {
    case 64: return launch_backward_one<T, ACC, 64>(m, dx, dw, s);
    case 128: return launch_backward_one<T, ACC, 128>(m, dx, dw, s);
    case 192: return launch_backward_one<T, ACC, 192>(m, dx, dw, s);
    default: return launch_backward_one<T, ACC, 256>(m, dx, dw, s);
  }
}

template <typename T>
int launch_backward(const BackwardProducts& p, int tile_n, int splits, int group_m, cudaStream_t s) {
  int dev = 0;
  cudaGetDevice(&dev);
  int* err = error_word(dev);
  CUtensorMap m[6];                                  // dy, w and dx of the one, dy, x and dw of the other
  int rc = make_tmap(&m[0], p.dy, p.n, p.t, p.ld_dy, BK, BM, p.dtype);
  if (rc == 0) rc = make_tmap(&m[1], p.w, p.k, p.n, p.ld_w, 64, BK, p.dtype);
  if (rc == 0) rc = make_tmap(&m[2], p.dx, p.k, p.t, p.ld_dx, 64, BM, p.dtype);
  if (rc == 0) rc = make_tmap(&m[3], p.dy, p.n, p.t, p.ld_dy, 64, BK, p.dtype);
  if (rc == 0) rc = make_tmap(&m[4], p.x, p.k, p.t, p.ld_x, 64, BK, p.dtype);
  if (rc == 0) rc = make_tmap(&m[5], p.dw, p.k, p.n, p.ld_dw, 64, BM, p.dtype);
  if (rc) return rc;
  const ClusterArgs dx = cluster_args(p.t, p.k, p.n, true, tile_n, splits, group_m, nullptr, nullptr, 0, err);
  const ClusterArgs dw = cluster_args(p.n, p.k, p.t, true, tile_n, splits, group_m, nullptr, p.row_sum, p.row_sum_add, err);
  return p.add_dw ? launch_backward_tile<T, true>(tile_n, m, dx, dw, s) : launch_backward_tile<T, false>(tile_n, m, dx, dw, s);
}

}  // namespace
}  // namespace gemm
}  // namespace ft
