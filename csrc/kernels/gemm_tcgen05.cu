// bf16 / fp16 GEMM on the 5th-generation tensor cores (sm_100a):
//   C[M,N] (=|+=) sum_k A(m,k) * B(n,k),  fp32 accumulation in tensor memory.
//
// Persistent, warp-specialised CTAs, one per SM:
//   warp 0      TMA producer: 128B-swizzled operand tiles into a 4-stage
//               shared-memory ring (cp.async.bulk.tensor, no cluster multicast)
//   warp 1      products: the whole warp runs the loop, an elected lane issues
//               tcgen05.mma 128x256x16 and tcgen05.commit; also owns
//               tensor-memory allocation
//   warps 2-5   epilogue: tcgen05.ld of the 128x256 fp32 accumulator, convert,
//               store (or add to C or to another matrix), from registers or by
//               way of shared memory (staged_epilogue)
// Two accumulator buffers (2 x 256 TMEM columns) let the epilogue of tile i
// overlap the main loop of tile i+1.  Tiles are walked in groups of 16 M-blocks
// so one wave of 148 CTAs shares operand tiles through L2.
//
// Operand layouts: an operand is "K-major" when the reduction index is the
// contiguous one in global memory and "MN-major" otherwise.  The three Linear
// GEMMs map to: forward (A K-major, B K-major), input gradient (A K-major,
// B MN-major), weight gradient (A MN-major, B MN-major) - no transposes are
// ever materialised.
//
// Replaces the cuBLAS calls a PyTorch model issues through F.linear on the
// reference's path.  Every mbarrier wait is bounded; on expiry the kernel
// records a code in a device error word, releases its tensor memory and returns.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "gemm2_kernel.cuh"
#include "gemm2_swiglu.cuh"
#include "gemm_cluster_host.h"
#include "gemm_host.h"

namespace {

using namespace ft;
using namespace ft::gemm;

// ------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

struct MapKey {
  const void* ptr;
  uint64_t inner, outer, ld;
  uint32_t box_inner, box_outer;
  int dtype;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && inner == o.inner && outer == o.outer && ld == o.ld &&
           box_inner == o.box_inner && box_outer == o.box_outer && dtype == o.dtype;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = std::hash<const void*>()(k.ptr);
    auto mix = [&](uint64_t v) { h ^= std::hash<uint64_t>()(v) + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2); };
    mix(k.inner); mix(k.outer); mix(k.ld); mix(k.box_inner); mix(k.box_outer); mix((uint64_t)k.dtype);
    return h;
  }
};

std::mutex g_map_mu;
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;

}  // namespace

namespace ft {
namespace gemm {

// 2-D row-major tensor [outer, inner] with row stride ld (elements), 128B swizzle.
// dtype: kBF16 / kF16 (2-byte elements) or kF32.
int make_tmap(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
              uint32_t box_inner, uint32_t box_outer, int dtype) {
  MapKey key{ptr, inner, outer, ld, box_inner, box_outer, dtype};
  {
    std::lock_guard<std::mutex> lk(g_map_mu);
    auto it = g_maps.find(key);
    if (it != g_maps.end()) { *out = it->second; return 0; }
  }
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -100;
  {
    // The driver entry point needs the primary context current in THIS thread; a
    // thread that has only used the runtime lazily (e.g. autograd's backward
    // thread) may not have bound it yet.  cudaSetDevice binds it; a cudaFree(nullptr), the older way, ends a
    // stream capture, and the output of a captured product is a new address each time.
    int dev = 0;
    cudaGetDevice(&dev);
    cudaSetDevice(dev);
  }
  const uint64_t esize = dtype == kF32 ? 4 : 2;
  if (((uintptr_t)ptr & 15) || ((ld * esize) & 15)) return -101;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * esize};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType dt = dtype == kF32    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : dtype == kBF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                  : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = fn(out, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    if (getenv("FLEXTRAIN_DEBUG")) fprintf(stderr, "cuTensorMapEncodeTiled -> %d ptr=%p inner=%llu outer=%llu ld=%llu box=%u,%u\n", (int)r, ptr, (unsigned long long)inner, (unsigned long long)outer, (unsigned long long)ld, box_inner, box_outer);
    return -102;
  }
  std::lock_guard<std::mutex> lk(g_map_mu);
  if (g_maps.size() > 8192) g_maps.clear();
  g_maps[key] = *out;
  return 0;
}

// One word per device, part of the library's image: the first launch may be captured into a graph, and
// an allocation or a memset may not.
__device__ int g_error_word;

int* error_word(int dev) {
  static std::atomic<int*> word[16];
  int* p = word[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_error_word);
    word[dev].store(p, std::memory_order_release);
  }
  return p;
}

int sm_count(int dev) {
  static std::atomic<int> count[16];
  int n = count[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    count[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace gemm
}  // namespace ft

namespace {

static_assert(SMEM_BYTES <= 232448 && P_SMEM_BYTES <= 232448 && P_SMEM_BYTES_GATHER <= 232448,
              "a GEMM kernel outgrew the 227 KB of dynamic shared memory of an SM");

// What the epilogue adds to the product, besides C itself (see GatherArgs): a matrix with its row
// stride, a row vector; nullptr each for none.  The tile width of the CTA-pair kernel.  And where it leaves the sums
// of A's rows (nullptr: nowhere).  The tiles that are divided over pairs, with the workspace for that.  The epilogue's way.
struct Addends { const void* matrix; int64_t ld; const void* bias; int tile_n; void* row_sum; int row_sum_add;
                 int split_tiles, split_pairs; void* workspace; int staged; };

// Columns of a CTA pair's tile: 256, 128 or 64.  Pairs take whole tiles, so the time is the number of
// rounds over the pairs times the time of a tile.  256 columns cost the least per column (A's bytes
// and the barriers are per tile: a tile takes about as long as its columns + 128), but 24 of them on 74
// pairs use a third of the machine, and a half as wide epilogue is half as long.  Widths between 128
// and 256 were measured and are not faster than 256 (12 x 10 tiles of 160 in two rounds: 79 us against 73
// for 12 x 7 of 256 in two).  All products of a 12-layer model of width 768 over 1024 tokens: 2.96 ms with
// 256, 2.40 ms with this rule.  fp32 results (the engine's fp32 gradient accumulators) stay at 256.
// "Columns + 128" is from before the product loops were run by whole warps; the clocks of a tile now are block_clocks'.  The rule
// is not always the best width with them, which matters for products of few tiles: those have a kernel of their own (cluster_plan).
int pair_tile_n(int M, int N, bool out32, int pairs) {
  if (pairs < 1) return P_BN;                        // no device: its launch is refused
  const int64_t mt = (M + P_BM - 1) / P_BM;
  auto cost = [&](int bn) {
    const int64_t tiles = mt * ((N + bn - 1) / bn);
    return (tiles + pairs - 1) / pairs * (bn + 128);
  };
  if (out32) return P_BN;
  int best = P_BN;
  for (int bn = 128; bn >= 64; bn /= 2)
    if (cost(bn) < cost(best)) best = bn;
  return best;
}

// How a product is divided over CTA pairs: the tile width, and how many tiles over how many pairs along the reduction
// (SplitWork; 0: none).
struct PairPlan { int tile_n, split_tiles, split_pairs; };

// Clocks of a k-block by tile width, of a divided tile's way through the workspace (the accumulators' two copies, the
// fence and the flags), and of adding a part where no whole tile follows under which that happens; parts of a tile at most.
// Measured, whole -> divided, us: 3000 x 1600 over 6400 63 -> 49, 2048 x 8192 over 8192 200 -> 183 and over 57344 1604 ->
// 1387, 1024 x 768 over 50304 145 -> 85, 4095 x 4096 over 32000 785 -> 710; 4096 x 4096 over 4096 93.5 -> 92.6.  With a
// cost of 3000 clocks short reductions were divided too and lost: 3000 x 4800 over 1600 58 -> 67, 4800 x 1600 over 3000 44 ->
// 48, 3000 x 1600 over 1600 23 -> 30.
constexpr double kSplitCost = 18000, kSplitAdd = 6000;
constexpr int kSplitParts = 6;
inline double block_clocks(int tile_n) { return tile_n == 256 ? 512 : tile_n == 128 ? 285 : 245; }

PairPlan pair_plan(int M, int N, int K, bool out32, int pairs) {
  const int mt = (M + P_BM - 1) / P_BM, kt = (K + BK - 1) / BK;
  PairPlan best{pair_tile_n(M, N, out32, pairs), 0, 0};
  if (pairs < 1) return best;
  auto tiles_of = [&](int bn) { return (int64_t)mt * ((N + bn - 1) / bn); };
  double least = 0.97 * ((tiles_of(best.tile_n) + pairs - 1) / pairs) * kt * block_clocks(best.tile_n);
  for (int bn = P_BN; bn >= (out32 ? P_BN : 64); bn /= 2) {
    const int64_t tiles = tiles_of(bn), whole = tiles / pairs, rest = tiles % pairs;
    if (rest == 0 || tiles > 1 << 20) continue;
    int64_t share = rest * kSplitParts < pairs ? rest * kSplitParts : pairs;
    if (share > rest * kt / (2 * SPLIT_MIN)) share = rest * kt / (2 * SPLIT_MIN);
    if (share <= rest) continue;
    const double run = (double)rest * kt / share, parts = (double)share / rest;       // k-blocks of a pair, pairs of a tile
    const double time = (whole * kt + run) * block_clocks(bn) + kSplitCost + (whole ? 0 : kSplitAdd * parts * bn / P_BN);
    if (time < least) { least = time; best = {bn, (int)rest, (int)share}; }
  }
  return best;
}

// Which products go to the cluster kernel (gemm_cluster.cuh), in what tiles: 16-bit results of aligned rows for which that is the
// fastest by the clocks below, tile_n 0: none.  A launch costs `start`; a pair works through its tiles one after another or two at
// a time, a k-block and a tile each taking what is stated.  Fitted to 570 products (192 to 4096 rows, widths of 256 to 16384,
// reductions of 256 to 16384, the three layouts; mean error 5 %, among neighbours in L2): chosen by it they take 0.77 of
// the persistent kernel's time, 0.75 with the best choice for each; us, before -> now: 256 x 256 over 256 3.8 -> 2.8, 2048 x 768 over
// 768 6.9 -> 4.7, 2048 x 2304 over 768 12.0 -> 7.7, 2048 x 768 over 3072 13.4 -> 10.6, 3072 x 768 += over 1024 9.2 -> 7.4.
// Not longer ones, nor operands beyond half of L2: the persistent kernel has twice the loads under way (192 x 12288 over 4096, 100 MB:
// 27.3 against 32.8, 1000 x 4096 over 4096 25.7 against 27.8); nor += in more than a round of 64 columns, of which the CTAs of a weight
// gradient load twice (1032 x 3776 over 1976 25.1 against 39.4).  Of 9 400 random products of 129 to 8192 rows and widths of 32 to
// 8192 that it takes, 22 are more than 3 % slower than they were; all together take 0.74 of the time.
struct ClusterPlan { int tile_n, splits; };
constexpr double kClusterLongest = 57000;            // 30 us
constexpr double kClusterBytes = 60e6;
// Pairs that run at a time: clusters of four CTAs leave SMs over in some groups of SMs (36 of them, 2198 x 504 over 3368: 18.2 -> 21.5).
inline int cluster_slots(int splits, int pairs) { return splits == 2 ? pairs - pairs / 12 : pairs; }
inline double cluster_clocks(int tn, int splits, bool acc, int tiles, int kt, int pairs) {
  const double start = tn == 192 ? 2850 : tn == 256 ? 2470 : splits == 2 ? 2090 : 2280;
  const double block = tn == 64 ? 270 : tn == 128 ? (splits == 2 ? 345 : acc ? 370 : 325) : tn == 192 ? (acc ? 570 : 490) : 575;
  const double tile = tn == 64 ? 2300 : tn == 128 ? (splits == 2 ? 5200 : acc ? 3200 : 2900) : tn == 192 ? (acc ? 3800 : 2900) : 3750;
  const int slots = cluster_slots(splits, pairs);
  return start + (tiles * splits + slots - 1) / slots * ((double)kt / splits * block + tile);
}
// The persistent kernel's, whole tiles.
inline double persistent_clocks(int tn, int tiles, int kt, int pairs) {
  const double start = tn == 64 ? 3230 : tn == 128 ? 4750 : 12600, block = tn == 64 ? 330 : tn == 128 ? 350 : 580,
               tile = tn == 64 ? 3200 : tn == 128 ? 4800 : 600;
  return start + (tiles + pairs - 1) / pairs * (kt * block + tile);
}

ClusterPlan cluster_plan(int M, int N, int K, bool acc, int widest, int pairs) {
  ClusterPlan best{0, 0};
  if (pairs < 1 || 2.0 * ((double)M * K + (double)N * K + (acc ? 2.0 : 1.0) * M * N) >= kClusterBytes) return best;
  const int mt = (M + P_BM - 1) / P_BM, kt = (K + BK - 1) / BK, tn0 = pair_tile_n(M, N, false, pairs);
  double least = 0.97 * persistent_clocks(tn0, mt * ((N + tn0 - 1) / tn0), kt, pairs);
  if (least > kClusterLongest) least = kClusterLongest;
  for (int tn = 64; tn <= widest; tn += 64) {
    if (tn == 64 && acc && mt * ((N + tn - 1) / tn) > pairs) continue;
    for (int splits = 1; splits <= (tn == 128 && kt >= 4 ? 2 : 1); ++splits) {
      const double t = cluster_clocks(tn, splits, acc, mt * ((N + tn - 1) / tn), kt, pairs);
      if (t < least) { least = t; best = {tn, splits}; }
    }
  }
  return best;
}

// Both products of a projection's backward pass in one launch (gemm_cluster_backward_kernel), dx of [t, k] over n and dw of [n, k] over
// t, in tiles and clusters alike for both; tile_n 0: one launch each is as good.  Their tiles are handed out longest first, so the
// time lies between that of their work spread evenly over the pairs and that of whole tiles one after another on each.
// One launch where that is to take 0.9 of two: chosen so 24 pairs of products took 0.79 of their time, us:
// t 256, n 768, k 256 6.8 -> 4.2; 1024, 768, 768 9.0 -> 6.0; 2048, 2304, 768 17.2 -> 13.2; 3000, 1600, 1600 46.7 -> 26.6.  Without a gain
// or not chosen: 1024, 3072, 768 13.9 -> 14.4; 4096, 1024, 1024 18.6 -> 18.5.
constexpr double kBackwardShare = 0.9, kBackwardBytes = 90e6;

double alone_clocks(int M, int N, int K, bool acc, int pairs) {
  const int mt = (M + P_BM - 1) / P_BM, kt = (K + BK - 1) / BK;
  const ClusterPlan p = cluster_plan(M, N, K, acc, P_BN, pairs);
  if (p.tile_n != 0) return cluster_clocks(p.tile_n, p.splits, acc, mt * ((N + p.tile_n - 1) / p.tile_n), kt, pairs);
  const int tn = pair_tile_n(M, N, false, pairs);
  return persistent_clocks(tn, mt * ((N + tn - 1) / tn), kt, pairs);
}

ClusterPlan backward_plan(int t, int n, int k, bool add_dw, bool sums, int pairs) {
  ClusterPlan best{0, 0};
  const double bytes = 2.0 * ((double)t * n + (double)(add_dw ? 3 : 2) * n * k + 2.0 * t * k);
  if (pairs < 1 || t <= 128 || n <= 128 || bytes >= kBackwardBytes) return best;
  double least = kBackwardShare * (alone_clocks(t, k, n, false, pairs) + alone_clocks(n, k, t, true, pairs));
  if (least > 2 * kClusterLongest) least = 2 * kClusterLongest;
  const int mt_dx = (t + P_BM - 1) / P_BM, mt_dw = (n + P_BM - 1) / P_BM, kt_dx = (n + BK - 1) / BK, kt_dw = (t + BK - 1) / BK;
  for (int tn = 64; tn <= (sums ? C_SUMS_TILE : P_BN); tn += 64) {
    for (int splits = 1; splits <= (tn == 128 && kt_dx >= 4 && kt_dw >= 4 ? 2 : 1); ++splits) {
      const int nt = (k + tn - 1) / tn;
      const double start = cluster_clocks(tn, splits, true, 0, 0, pairs);
      auto tile = [&](int kt) { return cluster_clocks(tn, splits, true, 1, kt, 2) - start; };
      double a = tile(kt_dx), b = tile(kt_dw);       // the longer and the shorter tiles
      int u = mt_dx * nt * splits, v = mt_dw * nt * splits;
      if (tn == 64 && u + v > pairs) continue;       // as in cluster_plan
      if (a < b) {
        const double c = a; a = b; b = c;
        const int w = u; u = v; v = w;
      }
      const int slots = cluster_slots(splits, pairs);
      double even = (u * a + v * b) / slots;
      if (even < a) even = a;
      double whole;                                  // the longer ones in rounds, the shorter ones where a round leaves room, then in rounds
      const int q = u / slots, r = u % slots, room = r ? (slots - r) * (int)(a / b) : 0;
      if (u + v <= slots) whole = a;
      else if (r == 0) whole = q * a + (v + slots - 1) / slots * b;
      else if (v <= room) whole = (q + 1) * a;
      else whole = (q + 1) * a + (v - room + slots - 1) / slots * b;
      const double time = start + 0.75 * whole + 0.25 * even;
      if (time < least) { least = time; best = {tn, splits}; }
    }
  }
  return best;
}

// Whether a 16-bit result whose rows are 16-byte aligned leaves by way of shared memory (epilogue_staged) rather than from
// registers (epilogue_tile).  It does where an addend has to be read and, from CTA pairs, where the last 32 columns are cut (from
// registers they would be single values for all rows).  Otherwise it is the longer way for one tile and the faster one beside products.  Staged against direct, speed with
// the direct epilogue of tiles of 256 columns = 1: 4096 x 4096 over 256 0.88, 512 0.97, 768 1.02, 1024 1.03; 16384 x 2048
// 0.91, 0.99, 1.05, 1.05; one tile a pair (2048 x 2048) 0.91, 0.94, 0.92, 0.94; with a bias 1.03 to 1.06 for all.  Narrower tiles:
// level.  Single-CTA kernel (tile_n 0), which has one tile a CTA: 64 x 4096 over 1024 0.83, 24 x 9600 over 64 0.76, 92 x 10640 over
// 1438 (cut) 0.90; with a bias 16 rows 0.94, 32 0.97, 64 1.02, 96 1.06.
bool staged_epilogue(int M, int N, int K, bool out32, bool addend, bool bias, int tile_n, int pairs) {
  if (out32 || N < 32 || N % 8) return false;
  if (addend) return true;
  if (tile_n == 0) return bias && M > 32;
  const int64_t tiles = (int64_t)((M + P_BM - 1) / P_BM) * ((N + tile_n - 1) / tile_n);
  return bias || N % 32 || tile_n < P_BN || (tiles > pairs && K >= 768);
}

constexpr int kWorkspaceWanted = -5;                 // ft_gemm_ws
int64_t split_bytes(const PairPlan& p) {
  return p.split_tiles == 0 ? 0 : (int64_t)p.split_pairs * (P_BM * p.tile_n * 4 + 8 * sizeof(uint64_t));
}

// A number no launch before had, from a start that differs between processes (the clock and where the library lies,
// mixed): what a workspace's memory held before is not taken for it.
uint64_t next_split_token() {
  static std::atomic<uint64_t> token{[] {
    uint64_t z = (uint64_t)std::chrono::steady_clock::now().time_since_epoch().count() ^
                 (uint64_t)reinterpret_cast<uintptr_t>(&g_map_mu) << 20;
    z = (z ^ z >> 30) * 0xbf58476d1ce4e5b9ULL;       // splitmix64's finish (Steele, Lea, Flood 2014)
    z = (z ^ z >> 27) * 0x94d049bb133111ebULL;
    return (z ^ z >> 31) | 1;
  }()};
  return token.fetch_add(2, std::memory_order_relaxed);
}

template <typename T, bool A_MN, bool B_MN>
int launch_mode(int mode, const CUtensorMap& ta, const CUtensorMap& tb, void* C, int64_t ldc, int M, int N,
                int K, int* err, int grid, cudaStream_t s, const Addends& add) {
  GatherArgs side{};
  side.add_src = add.matrix;
  side.add_ld = add.ld;
  side.bias = add.bias;
  side.staged = add.staged;
#define FT_LAUNCH(MODE)                                                                              \
  {                                                                                                  \
    auto kern = gemm_kernel<T, A_MN, B_MN, MODE>;                                                    \
    static DynamicSmem smem;                                                                         \
    smem.grant(kern, SMEM_BYTES);                                                                    \
    launch_overlapped(kern, grid, NUM_THREADS, add.staged ? SMEM_BYTES : SMEM_BYTES_DIRECT, s, 1,    \
                      overlap_product(M, N, K), ta, tb, C, ldc, M, N, K, err, side);                 \
  }
  switch (mode) {
    case kStore16: FT_LAUNCH(kStore16); break;
    case kStore32: FT_LAUNCH(kStore32); break;
    case kAcc16: FT_LAUNCH(kAcc16); break;
    case kAcc32: FT_LAUNCH(kAcc32); break;
    case kAcc16Cut: FT_LAUNCH(kAcc16Cut); break;
    default: return -3;
  }
#undef FT_LAUNCH
  return 0;
}

// ---- CTA-pair kernel (cluster of 2)
// Row blocks per group of the CTA-pair kernel's tile walk (FLEXTRAIN_GEMM_GROUP_M, default 16).
int pair_group_m() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("FLEXTRAIN_GEMM_GROUP_M");
    v = e ? atoi(e) : GROUP_M;
    if (v < 1) v = GROUP_M;
  }
  return v;
}

template <typename T, bool A_MN, bool B_MN, int MODE, int TN>
int launch_pair_one(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int64_t ldc, int M, int N, int K,
                    int* err, int grid, cudaStream_t s, const Addends& add) {
  auto kern = gemm_pair_kernel<T, A_MN, B_MN, MODE, false, TN>;
  static DynamicSmem smem;
  smem.grant(kern, P_SMEM_BYTES);
  GatherArgs none{};
  none.group_m = pair_group_m();
  none.add_src = add.matrix;
  none.add_ld = add.ld;
  none.bias = add.bias;
  none.staged = add.staged;
  none.row_sum = add.row_sum;
  none.row_sum_add = add.row_sum_add;
  if (add.split_tiles > 0) {
    none.split_tiles = add.split_tiles;
    none.split_pairs = add.split_pairs;
    none.split_token = next_split_token();
    none.split_sums = static_cast<float*>(add.workspace);
    none.split_flags = reinterpret_cast<uint64_t*>(none.split_sums + (int64_t)add.split_pairs * P_BM * TN);
  }
  const bool slots = add.staged || add.split_tiles > 0 || add.row_sum != nullptr;
  cudaError_t e = launch_overlapped(kern, grid, NUM_THREADS, slots ? P_SMEM_BYTES : P_SMEM_BYTES_DIRECT, s, 2,
                                    overlap_product(M, N, K), ta, tb, C, ldc, M, N, K, err, none);
  return e == cudaSuccess ? 0 : (int)e;
}

template <typename T, bool A_MN, bool B_MN>
int launch_pair_mode(int mode, const CUtensorMap& ta, const CUtensorMap& tb, void* C, int64_t ldc, int M,
                     int N, int K, int* err, int grid, cudaStream_t s, const Addends& add) {
#define FT_PAIR(MODE, TN) return launch_pair_one<T, A_MN, B_MN, MODE, TN>(ta, tb, C, ldc, M, N, K, err, grid, s, add)
  switch (mode) {
    case kStore16:
      if (add.tile_n == 64) FT_PAIR(kStore16, 64);
      if (add.tile_n == 128) FT_PAIR(kStore16, 128);
      FT_PAIR(kStore16, 256);
    case kAcc16:
      if (add.tile_n == 64) FT_PAIR(kAcc16, 64);
      if (add.tile_n == 128) FT_PAIR(kAcc16, 128);
      FT_PAIR(kAcc16, 256);
    case kStore32: FT_PAIR(kStore32, 256);
    case kAcc32: FT_PAIR(kAcc32, 256);
    case kAcc16Cut:
      if (add.tile_n == 64) FT_PAIR(kAcc16Cut, 64);
      if (add.tile_n == 128) FT_PAIR(kAcc16Cut, 128);
      FT_PAIR(kAcc16Cut, 256);
    default: return -3;
  }
#undef FT_PAIR
}

template <typename T>
int launch_pair(int a_mn, int b_mn, int mode, const CUtensorMap& ta, const CUtensorMap& tb, void* C,
                int64_t ldc, int M, int N, int K, int* err, int grid, cudaStream_t s, const Addends& add) {
  if (!a_mn && !b_mn) return launch_pair_mode<T, false, false>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  if (!a_mn && b_mn) return launch_pair_mode<T, false, true>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  if (a_mn && b_mn) return launch_pair_mode<T, true, true>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  return launch_pair_mode<T, true, false>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
}

int g_use_pair = -1;   // -1: read FLEXTRAIN_GEMM_PAIR on first use

bool pair_wanted() {
  if (g_use_pair < 0) {
    const char* e = getenv("FLEXTRAIN_GEMM_PAIR");
    g_use_pair = e ? atoi(e) : 1;
  }
  return g_use_pair != 0;
}

template <typename T>
int launch_pair_swiglu(const CUtensorMap& ta, const CUtensorMap& tb, void* act, int64_t ld_act, void* gu,
                       int64_t ld_gu, int M, int F, int K, int* err, int grid, cudaStream_t s) {
  auto kern = gemm_pair_swiglu_kernel<T>;
  static DynamicSmem smem;
  smem.grant(kern, P_SMEM_BYTES);
  cudaError_t e = launch_overlapped(kern, grid, NUM_THREADS, P_SMEM_BYTES, s, 2, overlap_product(M, 2 * (int64_t)F, K), ta,
                                    tb, act, ld_act, gu, ld_gu, M, F,
                                    K, err);
  return e == cudaSuccess ? 0 : (int)e;
}

template <typename T>
int launch_layout(int a_mn, int b_mn, int mode, const CUtensorMap& ta, const CUtensorMap& tb, void* C,
                  int64_t ldc, int M, int N, int K, int* err, int grid, cudaStream_t s, const Addends& add) {
  if (!a_mn && !b_mn) return launch_mode<T, false, false>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  if (!a_mn && b_mn) return launch_mode<T, false, true>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  if (a_mn && b_mn) return launch_mode<T, true, true>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
  return launch_mode<T, true, false>(mode, ta, tb, C, ldc, M, N, K, err, grid, s, add);
}

}  // namespace

namespace {

int gemm_launch(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
                int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
                int ab_dtype, void* row_sum, int row_sum_add, void* workspace,
                int64_t workspace_bytes, cudaStream_t stream);

}  // namespace

extern "C" {

int ft_gemm_bias(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
                 int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
                 int ab_dtype, cudaStream_t stream);
int ft_gemm_ws(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
               int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
               int ab_dtype, void* workspace, int64_t workspace_bytes, cudaStream_t stream);

// Columns of an output tile of the CTA-pair kernel for C of M x N (c_dtype 0: fp32) on `pairs` CTA pairs: the
// rule, for its tests.
int ft_gemm_tile_n(int M, int N, int c_dtype, int pairs) { return pair_tile_n(M, N, c_dtype == kF32, pairs); }

// C = A B + R with fp32 accumulation, R a matrix of C's type and shape (row stride ldr).  R = nullptr gives
// C = A B (accumulate 0) or C += A B (accumulate 1).  R may not overlap C unless it is C.
//   A: K-major -> stored [M,K] (row stride lda); MN-major (a_mn=1) -> stored [K,M].
//   B: K-major -> stored [N,K] (row stride ldb); MN-major (b_mn=1) -> stored [K,N].
//   C: [M,N], row stride ldc, dtype c_dtype (same 16-bit type as A/B, or fp32).
// Returns 0, a negative argument error, or a positive CUDA error code.
int ft_gemm_add(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C,
                int64_t ldc, int c_dtype, int accumulate, const void* R, int64_t ldr, int M, int N, int K,
                int ab_dtype, cudaStream_t stream) {
  return ft_gemm_bias(A, a_mn, lda, B, b_mn, ldb, C, ldc, c_dtype, accumulate, R, ldr, nullptr, M, N, K, ab_dtype,
                      stream);
}

// As ft_gemm_add, and a row vector `bias` (N values of C's type, N a multiple of 8, 16-byte aligned;
// nullptr: none) is added to every row before the one rounding of the result.  C is 16-bit and both
// operands are K-major then.
int ft_gemm_bias(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C,
                 int64_t ldc, int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N,
                 int K, int ab_dtype, cudaStream_t stream) {
  return ft_gemm_ws(A, a_mn, lda, B, b_mn, ldb, C, ldc, c_dtype, accumulate, R, ldr, bias, M, N, K, ab_dtype, nullptr,
                    0, stream);
}

// As ft_gemm_bias, with a workspace of the caller's of at least ft_gemm_ws_bytes(...) bytes that nothing else uses
// until the product is done; its contents need no preparation.  With less (or nullptr) tiles are not divided.  With
// workspace_bytes -1 a product that would be divided is not launched and the answer is kWorkspaceWanted: callers ask and launch
// in one call, because most products are not divided and small ones are bound by the host (a question of its own
// took ctypes 1.4 of 6.2 us).
int ft_gemm_ws(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
               int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
               int ab_dtype, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  return gemm_launch(A, a_mn, lda, B, b_mn, ldb, C, ldc, c_dtype, accumulate, R, ldr, bias, M, N, K, ab_dtype, nullptr,
                     0, workspace, workspace_bytes, stream);
}

// The first of those calls without the arguments that most products leave empty, a tenth of the time ctypes takes.
int ft_gemm_try(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
                int c_dtype, int accumulate, int M, int N, int K, int ab_dtype, cudaStream_t stream) {
  return gemm_launch(A, a_mn, lda, B, b_mn, ldb, C, ldc, c_dtype, accumulate, nullptr, 0, nullptr, M, N, K, ab_dtype,
                     nullptr, 0, nullptr, -1, stream);
}

// Bytes of workspace (16-byte aligned) with which ft_gemm_ws divides tiles of this product over CTA pairs on the
// current device; 0 where it would not.
int64_t ft_gemm_ws_bytes(int M, int N, int K, int c_dtype) {
  if (M <= 128 || N <= 0 || K <= 0 || !pair_wanted()) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  return split_bytes(pair_plan(M, N, K, c_dtype == kF32, sm_count(dev) / 2));
}

// The plan itself on `pairs` CTA pairs, for its tests: tile width | divided tiles << 16 | pairs they are divided over << 32.
int64_t ft_gemm_split_plan(int M, int N, int K, int c_dtype, int pairs) {
  const PairPlan p = pair_plan(M, N, K, c_dtype == kF32, pairs);
  return p.tile_n | (int64_t)p.split_tiles << 16 | (int64_t)p.split_pairs << 32;
}

// The cluster kernel's plan on `pairs` CTA pairs, for its tests: tile width | pairs a cluster << 16; 0: not its product.
// Bit 1 of `accumulate`: with the sums of A's rows.
int ft_gemm_cluster_plan(int M, int N, int K, int accumulate, int pairs) {
  const ClusterPlan p = cluster_plan(M, N, K, accumulate & 1, accumulate & 2 ? C_SUMS_TILE : P_BN, pairs);
  return p.tile_n | p.splits << 16;
}

// Whether the epilogue goes by way of shared memory, on `pairs` CTA pairs (the rule, for its tests).
int ft_gemm_staged(int M, int N, int K, int c_dtype, int accumulate, int bias, int pairs) {
  return staged_epilogue(M, N, K, c_dtype == kF32, accumulate, bias, M > 128 ? pair_tile_n(M, N, c_dtype == kF32, pairs) : 0, pairs);
}

// Gradients of a biased projection: dw[N, K] (=|+=) sum_t dy(t, n) x(t, k) and db[N] (=|+=) sum_t dy(t, n), from
// dy [T, N] and x [T, K] of the 16-bit type `dtype`, which dw and db have too.  -4 where the product does not sum on
// the way (tiles of 256 columns leave no accumulator for it, N <= 128 has a kernel of its own): the caller then sums itself.
int ft_gemm_dw_db(const void* dy, int64_t ld_dy, const void* x, int64_t ld_x, void* dw, int64_t ld_dw, int add_dw,
                  void* db, int add_db, int T, int N, int K, int dtype, cudaStream_t stream) {
  if (T <= 0 || N <= 0 || K <= 0) return -4;
  if (dtype != kBF16 && dtype != kF16) return -1;
  int dev = 0;
  cudaGetDevice(&dev);
  const int pairs = sm_count(dev) / 2;
  if (N <= 128 || !pair_wanted() ||
      (pair_tile_n(N, K, false, pairs) > 128 && cluster_plan(N, K, T, add_dw != 0, C_SUMS_TILE, pairs).tile_n == 0))
    return -4;
  return gemm_launch(dy, 1, ld_dy, x, 1, ld_x, dw, ld_dw, dtype, add_dw, nullptr, 0, nullptr, N, K, T, dtype, db, add_db,
                     nullptr, 0, stream);
}

// dx[t, k] = dy w and dw[n, k] (=|+=) dy^T x, with db[n] (=|+=) the column sums of dy where db is given, in one launch: dy [t, n], w [n, k]
// and x [t, k] of the 16-bit type `dtype`, which the results have too.  -4 where two launches are as good, or rows are not 16-byte
// aligned: nothing has been launched.
int ft_gemm_backward(const void* dy, int64_t ld_dy, const void* w, int64_t ld_w, const void* x, int64_t ld_x, void* dx,
                     int64_t ld_dx, void* dw, int64_t ld_dw, int add_dw, void* db, int add_db, int t, int n, int k, int dtype,
                     cudaStream_t stream) {
  if (t <= 0 || n <= 0 || k <= 0 || !pair_wanted()) return -4;
  if (dtype != kBF16 && dtype != kF16) return -1;
  if ((k | ld_dy | ld_w | ld_x | ld_dx | ld_dw) % 8 || !aligned16(dy) || !aligned16(w) || !aligned16(x) || !aligned16(dx) || !aligned16(dw))
    return -4;
  int dev = 0;
  cudaGetDevice(&dev);
  const ClusterPlan plan = backward_plan(t, n, k, add_dw != 0, db != nullptr, sm_count(dev) / 2);
  if (plan.tile_n == 0) return -4;
  const BackwardProducts p{dy, w, x, dx, dw, db, ld_dy, ld_w, ld_x, ld_dx, ld_dw, t, n, k, add_dw, add_db, dtype};
  const int rc = dtype == kBF16 ? launch_backward<__nv_bfloat16>(p, plan.tile_n, plan.splits, pair_group_m(), stream)
                                : launch_backward<__half>(p, plan.tile_n, plan.splits, pair_group_m(), stream);
  if (rc) return rc;
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// Its plan on `pairs` CTA pairs, for its tests: tile width | pairs a cluster << 16; 0: two launches.
int ft_gemm_backward_plan(int t, int n, int k, int add_dw, int sums, int pairs) {
  const ClusterPlan p = backward_plan(t, n, k, add_dw != 0, sums != 0, pairs);
  return p.tile_n | p.splits << 16;
}

}  // extern "C"

namespace {

int gemm_launch(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
                int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
                int ab_dtype, void* row_sum, int row_sum_add, void* workspace,
                int64_t workspace_bytes, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (R != nullptr) accumulate = 1;
  if (ab_dtype != kBF16 && ab_dtype != kF16) return -1;
  if (c_dtype != kF32 && c_dtype != ab_dtype) return -2;
  if (bias != nullptr && (a_mn || b_mn || c_dtype == kF32 || N % 8 || (reinterpret_cast<uintptr_t>(bias) & 15))) return -2;
  // The epilogue's 16-byte accesses go by the row strides (store_chunk); the pointers are checked here.
  const int align = c_dtype == kF32 ? 4 : 8;
  const bool vec = ldc % align == 0 && (R == nullptr || ldr % align == 0) && N >= (accumulate ? 16 : 32);
  if (vec && ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(R)) & 15)) return -2;
  int dev = 0;
  cudaGetDevice(&dev);
  int* err = error_word(dev);
  CUtensorMap ta, tb;
  int rc;
  const bool use_pair = pair_wanted();
  // The pair kernel's tile is 256 rows tall: below that half of it would be padding.
  const bool pair = use_pair && M > 128;
  PairPlan plan{BN, 0, 0};
  // whole 16-byte units only: a TMA store writes the unit that the matrix's edge cuts to its end
  const bool rows16 = c_dtype != kF32 && N % 8 == 0 && ldc % 8 == 0 && (R == nullptr || ldr % 8 == 0) &&
                      !((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(R)) & 15);
  if (pair && rows16 && !(a_mn && !b_mn)) {
    const ClusterPlan cp = cluster_plan(M, N, K, accumulate != 0, row_sum != nullptr ? C_SUMS_TILE : P_BN, sm_count(dev) / 2);
    if (cp.tile_n != 0) {
      const ClusterProduct p{A, B, C, accumulate ? (R != nullptr ? R : C) : nullptr, bias, lda, ldb, ldc, R != nullptr ? ldr : ldc,
                             a_mn, b_mn, M, N, K, ab_dtype, row_sum, row_sum_add};
      rc = ab_dtype == kBF16 ? launch_cluster<__nv_bfloat16>(p, cp.tile_n, cp.splits, pair_group_m(), stream)
                             : launch_cluster<__half>(p, cp.tile_n, cp.splits, pair_group_m(), stream);
      if (rc) return rc;
      FT_LAUNCHED(1);
      FT_CUDA_RETURN_IF_ERROR();
      return 0;
    }
  }
  if (row_sum != nullptr && pair_tile_n(M, N, false, sm_count(dev) / 2) > 128) return -4;
  if (pair) {
    plan = {pair_tile_n(M, N, c_dtype == kF32, sm_count(dev) / 2), 0, 0};
    if (workspace != nullptr || workspace_bytes < 0) {
      const PairPlan p = pair_plan(M, N, K, c_dtype == kF32, sm_count(dev) / 2);
      if (workspace_bytes < 0 && p.split_tiles > 0) return kWorkspaceWanted;
      if (split_bytes(p) <= workspace_bytes && !(reinterpret_cast<uintptr_t>(workspace) & 15)) plan = p;
    }
  }
  const int tile_n = plan.tile_n;
  const int b_box = pair ? tile_n / 2 : BN;       // rows of B one CTA stages per k-block
  const int staged = ldc % 8 == 0 && (R == nullptr || ldr % 8 == 0) &&
                     staged_epilogue(M, N, K, c_dtype == kF32, accumulate, bias != nullptr, pair ? tile_n : 0, sm_count(dev) / 2);
  const Addends add{R, ldr, bias, tile_n, row_sum, row_sum_add, plan.split_tiles, plan.split_pairs, workspace, staged};
  if (a_mn) rc = make_tmap(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, BK, ab_dtype);
  else rc = make_tmap(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, BM, ab_dtype);
  if (rc) return rc;
  if (b_mn) rc = make_tmap(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, BK, ab_dtype);
  else rc = make_tmap(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, b_box, ab_dtype);
  if (rc) return rc;
  const bool cut = N % 8 && N >= 16 && ldc % 8 == 0 && (R == nullptr || ldr % 8 == 0) && row_sum == nullptr;
  const int mode = c_dtype == kF32 ? (accumulate ? kAcc32 : kStore32) : accumulate ? (cut ? kAcc16Cut : kAcc16) : kStore16;
  if (pair) {
    const int tiles = ((M + P_BM - 1) / P_BM) * ((N + tile_n - 1) / tile_n);
    const int pairs = sm_count(dev) / 2;
    const int grid = 2 * (tiles >= pairs ? pairs : tiles > plan.split_pairs ? tiles : plan.split_pairs);
    if (ab_dtype == kBF16)
      rc = launch_pair<__nv_bfloat16>(a_mn, b_mn, mode, ta, tb, C, ldc, M, N, K, err, grid, stream, add);
    else
      rc = launch_pair<__half>(a_mn, b_mn, mode, ta, tb, C, ldc, M, N, K, err, grid, stream, add);
  } else {
    const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    const int grid = tiles < sm_count(dev) ? tiles : sm_count(dev);
    if (ab_dtype == kBF16)
      rc = launch_layout<__nv_bfloat16>(a_mn, b_mn, mode, ta, tb, C, ldc, M, N, K, err, grid, stream, add);
    else
      rc = launch_layout<__half>(a_mn, b_mn, mode, ta, tb, C, ldc, M, N, K, err, grid, stream, add);
  }
  if (rc) return rc;
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

}  // namespace

extern "C" {

// C[M,N] (=|+=) A x B^T-like product: ft_gemm_add without R.
int ft_gemm(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C,
            int64_t ldc, int c_dtype, int accumulate, int M, int N, int K, int ab_dtype,
            cudaStream_t stream) {
  return ft_gemm_add(A, a_mn, lda, B, b_mn, ldb, C, ldc, c_dtype, accumulate, nullptr, 0, M, N, K, ab_dtype,
                     stream);
}

// act[M,F] = silu(X Wg^T) * (X Wu^T) with W = [Wg ; Wu] stored [2F, K] (row stride ldw), X stored
// [M, K] (row stride ldx); gu (optional, [M, 2F], row stride ld_gu) receives the two projections
// as the unfused path would have stored them.  Returns -4 when the shape is not covered (F not a
// multiple of 128, fewer than 129 rows): the caller then runs ft_gemm + the activation kernel.
int ft_gemm_swiglu(const void* X, int64_t ldx, const void* W, int64_t ldw, void* act, int64_t ld_act,
                   void* gu, int64_t ld_gu, int M, int F, int K, int dtype, cudaStream_t stream) {
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if (dtype != kBF16 && dtype != kF16) return -1;
  if (F % 128 || M <= 128) return -4;
  int dev = 0;
  cudaGetDevice(&dev);
  int* err = error_word(dev);
  CUtensorMap ta, tb;
  int rc = make_tmap(&ta, X, (uint64_t)K, (uint64_t)M, (uint64_t)ldx, BK, BM, dtype);
  if (rc) return rc;
  rc = make_tmap(&tb, W, (uint64_t)K, (uint64_t)(2 * F), (uint64_t)ldw, BK, 128, dtype);
  if (rc) return rc;
  const int tiles = ((M + P_BM - 1) / P_BM) * (F / 128);
  const int pairs = sm_count(dev) / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  if (dtype == kBF16)
    rc = launch_pair_swiglu<__nv_bfloat16>(ta, tb, act, ld_act, gu, ld_gu, M, F, K, err, grid, stream);
  else
    rc = launch_pair_swiglu<__half>(ta, tb, act, ld_act, gu, ld_gu, M, F, K, err, grid, stream);
  if (rc) return rc;
  FT_LAUNCHED(1);
  FT_CUDA_RETURN_IF_ERROR();
  return 0;
}

// Selects the CTA-pair kernel (1) or the single-CTA kernel (0) for later ft_gemm calls.
void ft_gemm_set_pair(int on) { g_use_pair = on ? 1 : 0; }
int ft_gemm_get_pair() { return g_use_pair > 0 ? 1 : 0; }

// Reads (and clears) the device error word: 0 = no bounded wait ever expired.
// Synchronises the device; meant for tests and health checks.
int ft_gemm_error() {
  int dev = 0;
  cudaGetDevice(&dev);
  int* err = error_word(dev);
  int host = 0;
  if (cudaMemcpy(&host, err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (host) cudaMemset(err, 0, sizeof(int));
  return host;
}

}  // extern "C"
