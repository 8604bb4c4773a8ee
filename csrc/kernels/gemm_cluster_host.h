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
  const int kt = (p.K + BK - 1) / BK, stages = cluster_stages(tile_n, p.b_mn);
  const ClusterArgs args{p.M, p.N, p.K, splits, stages, kt % stages, (p.M + P_BM - 1) / P_BM, (p.N + tile_n - 1) / tile_n, kt,
                         group_m, p.bias, p.row_sum, p.row_sum_add, error_word(dev)};
#define FT_CLUSTER(A_MN, B_MN)                                                                                   \
  return p.R != nullptr ? launch_cluster_tile<T, A_MN, B_MN, true>(tile_n, ta, tb, tc, tr, args, s)       \
                        : launch_cluster_tile<T, A_MN, B_MN, false>(tile_n, ta, tb, tc, tr, args, s)
  if (!p.a_mn && !p.b_mn) FT_CLUSTER(false, false);
  if (!p.a_mn) FT_CLUSTER(false, true);
  if (p.b_mn) FT_CLUSTER(true, true);
#undef FT_CLUSTER
  return -4;
}

}  // namespace
}  // namespace gemm
}  // namespace ft
