// Launches of the FMA products (cgt_product.h): which kernel, which tile, how K is split.
#include <algorithm>
#include "products.h"
#include "runtime.h"

namespace cgtb {
using namespace tile;

namespace {

struct Split {
  int bt, cluster, nsplit;
};
// Fitted to measured times (microseconds; slices of 256 bytes of k per row): a slice takes a 32 x 32 tile 0.62 and a
// 64 x 64 tile 2.1, times the blocks per SM when the grid exceeds one per SM; a fold through a cluster costs 1.2 plus
// 0.1 per block. 128 x 256 x 784: 32 x 32 tiles in clusters of four, 6.4 us (one block per tile: 11.2); 1024^3: 57 us.
// What a cluster of eight leaves longer than eight slices is cut over several clusters, whose slabs a second kernel adds.
template <typename T>
Split choose_split(long P, long M, long N, long K) {
  const long slices = cgtb_ceil_div(K, Shape<T, 32>::KT);
  Split best = {32, 1, 1};
  double best_t = 1e30;
  for (int bt = 32; bt <= 64; bt += 32) {
    const double tiles = (double)cgtb_ceil_div(M, bt) * cgtb_ceil_div(N, bt) * P, slice_us = bt == 32 ? 0.62 : 2.1;
    for (int c = 1; c <= 8; c *= 2) {
      if (c > slices) break;
      long own = cgtb_ceil_div(slices, c);
      int ns = 1;
      if (c == 8 && own > 8) {
        ns = (int)std::min<long>(cgtb_ceil_div(own, 4), std::max<long>(1, (long)(rt().sm_count / (tiles * c))));
        own = cgtb_ceil_div(own, ns);
      }
      const double load = std::max(1.0, tiles * c * ns / rt().sm_count);
      const double t = own * slice_us * load + (c > 1 ? 1.2 + 0.1 * c : 0.0) + (ns > 1 ? 2.5 : 0.0);
      if (t < best_t) {
        best_t = t;
        best = {bt, c, ns};
      }
    }
  }
  return best;
}

// One warp per output suits few outputs, or operands that both run along K in memory (its lanes read along K); few rows
// against a matrix stored along n have a kernel of their own.
bool warp_per_output(int tA, int tB, long M, long N) { return (M > 8 || tB) && (M * N <= 2048 || (!tA && tB)); }
bool small_shape(long P, long M, long N, long K) { return M * N <= 65536 && K <= 2048 && M * N * K <= (1L << 24) && P <= 65535; }

template <typename T>
struct Planned {
  Plan plan;
  Split split;
};
// allow_small: the kernels with one warp per output may be chosen (float only)
template <typename T>
Planned<T> plan_product(int tA, int tB, long P, long M, long N, long K, bool allow_small) {
  Planned<T> r = {};
  r.split = {32, 1, 1};
  r.plan.cluster = 1;
  if (allow_small && sizeof(T) == 4 && warp_per_output(tA, tB, M, N) && small_shape(P, M, N, K)) {
    const int lanes = K >= 128 ? 32 : (K >= 32 ? 8 : 1);
    if (lanes == 32 && !tA && tB && M % 4 == 0 && N % 4 == 0 && M * N >= 1024) {
      r.plan.variant = kSmallNT;
      r.plan.grid = dim3((unsigned)cgtb_ceil_div((M / 4) * (N / 4) * 32, 256), (unsigned)P);
    } else {
      r.plan.variant = kSmall | lanes;
      r.plan.grid = dim3((unsigned)cgtb_ceil_div(M * N * lanes, 256), (unsigned)P);
    }
    return r;
  }
  if (M <= 8 && !tB && K > 0) {
    const long blocks = cgtb_ceil_div(N, 32);
    int c = 1;
    while (c < 8 && cgtb_ceil_div(K, 2 * c) >= 64 && blocks * P * c < rt().sm_count) c *= 2;
    r.split.cluster = r.plan.cluster = c;
    r.plan.variant = kRows | (M == 1 ? 1 : (M <= 4 ? 4 : 8));
    r.plan.grid = dim3((unsigned)blocks, 1, (unsigned)(P * c));
    return r;
  }
  r.split = choose_split<T>(P, M, N, K);
  r.plan.cluster = r.split.cluster;
  r.plan.variant = (r.split.nsplit > 1 ? kTilesFold : kTiles) | (r.split.bt == 64 ? 1 : 0) | (!tA ? 2 : 0) | (tB ? 4 : 0);
  r.plan.grid = dim3((unsigned)(cgtb_ceil_div(M, r.split.bt) * cgtb_ceil_div(N, r.split.bt)), 1, (unsigned)(P * r.split.cluster * r.split.nsplit));
  return r;
}

template <typename T>
bool loads_vec(const T* p, long ld, long stride, long P) {
  constexpr int VW = 16 / (int)sizeof(T);
  return ((uintptr_t)p & 15) == 0 && ld % VW == 0 && (P <= 1 || stride % VW == 0);
}

template <typename T>
cudaError_t launch_tiles_any(const Plan& p, const Args<T>& a, cudaStream_t st) {
  const Store<T> e;
  switch (p.variant & 7) {
    case 0: return launch_tiles<T, 0>(p, a, e, st);
    case 1: return launch_tiles<T, 1>(p, a, e, st);
    case 2: return launch_tiles<T, 2>(p, a, e, st);
    case 3: return launch_tiles<T, 3>(p, a, e, st);
    case 4: return launch_tiles<T, 4>(p, a, e, st);
    case 5: return launch_tiles<T, 5>(p, a, e, st);
    case 6: return launch_tiles<T, 6>(p, a, e, st);
    default: return launch_tiles<T, 7>(p, a, e, st);
  }
}
template <typename T>
cudaError_t launch_any(const Plan& p, const Args<T>& a, cudaStream_t st) {
  const Store<T> e;
  if (p.variant & (kTiles | kTilesFold)) return launch_tiles_any<T>(p, a, st);
  switch (p.variant) {
    case kRows | 1: return launch_single<T, kRows | 1>(p, a, e, st);
    case kRows | 4: return launch_single<T, kRows | 4>(p, a, e, st);
    case kRows | 8: return launch_single<T, kRows | 8>(p, a, e, st);
  }
  if constexpr (sizeof(T) == 4) {
    switch (p.variant) {
      case kSmallNT: return launch_single<T, kSmallNT>(p, a, e, st);
      case kSmall | 1: return launch_single<T, kSmall | 1>(p, a, e, st);
      case kSmall | 8: return launch_single<T, kSmall | 8>(p, a, e, st);
      case kSmall | 32: return launch_single<T, kSmall | 32>(p, a, e, st);
    }
  }
  return cudaErrorInvalidValue;
}

template <typename T>
int run_product(const Product<T>& q, const Planned<T>& pl) {
  const Plan& p = pl.plan;
  if (p.grid.x == 0 || p.grid.z > 65535 || p.grid.y > 65535 || cgtb_ceil_div(q.M, 32) * cgtb_ceil_div(q.N, 32) > 2147483647L)
    return fail("product: grid too large (M=%ld N=%ld, %ld batches)", q.M, q.N, q.P);
  if (q.chain && q.chain->variant != p.variant) return -1;
  Args<T> a = {};
  a.M = q.M;
  a.N = q.N;
  a.K = q.K;
  a.A = q.A;
  a.B = q.B;
  a.lda = q.lda;
  a.ldb = q.ldb;
  a.stride_a = q.strideA;
  a.stride_b = q.strideB;
  a.C = q.C;
  a.ldc = q.ldc;
  a.stride_c = q.strideC;
  a.tA = q.tA;
  a.tB = q.tB;
  a.sums = q.sums;
  a.vec_a = loads_vec(q.A, q.lda, q.strideA, q.P);
  a.vec_b = loads_vec(q.B, q.ldb, q.strideB, q.P);
  a.cluster = pl.split.cluster;
  a.nsplit = pl.split.nsplit;
  a.tiles_n = (int)cgtb_ceil_div(q.N, pl.split.bt);
  const long parts = (long)a.cluster * a.nsplit, KT = (p.variant & (kTiles | kTilesFold)) ? Shape<T, 32>::KT : 1;
  a.kchunk = std::max<long>(KT, cgtb_ceil_div(cgtb_ceil_div(q.K, parts), KT) * KT);
  cudaStream_t st = rt().stream;
  cudaError_t e = cudaSuccess;
  auto chain = [&](const void* part) {
    const Chain& c = *q.chain;
    return c.launch(&p, &a, part, pl.split.nsplit, c.in, c.bk, c.bi, c.out, (void*)st) ? cudaErrorUnknown : cudaSuccess;
  };
  if (a.nsplit > 1) {
    T* part = (T*)scratch((size_t)q.P * a.nsplit * q.M * q.N * sizeof(T));
    if (!part) return 1;
    a.C = part;
    e = launch_tiles_any<T>(p, a, st);
    a.C = q.C;
    if (e == cudaSuccess) e = q.chain ? chain(part) : launch_fold<T>(part, a.nsplit, a, q.P, Store<T>(), st);
    g_kernel_launches.fetch_add(2, std::memory_order_relaxed);
  } else {
    e = q.chain ? chain(nullptr) : launch_any<T>(p, a, st);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail("product launch failed: %s", cudaGetErrorString(e));
  }
  return 0;
}

template <typename T>
int product_fma_t(const Product<T>& q, bool tiles_only) {
  if (q.P <= 0 || q.M <= 0 || q.N <= 0) return 0;
  return run_product<T>(q, plan_product<T>(q.tA, q.tB, q.P, q.M, q.N, q.K, !tiles_only && !q.sums.bias && !q.sums.addend));
}
}  // namespace

bool product_is_fma(int tA, int tB, long P, long M, long N, long K) {
  if (warp_per_output(tA, tB, M, N) && small_shape(P, M, N, K)) return true;
  if (P > 65535) return false;  // one grid layer per product
  return M * N * K <= (1L << 25) || P * M * N * K <= (1L << 26);
}
int product_fma(const Product<float>& q, bool tiles_only) { return product_fma_t(q, tiles_only); }
int product_fma(const Product<double>& q, bool tiles_only) { return product_fma_t(q, tiles_only); }
int product_small(const Product<float>& q) {
  if (q.P <= 0 || q.M <= 0 || q.N <= 0) return 0;
  if (!small_shape(q.P, q.M, q.N, q.K)) return -1;
  const int lanes = q.K >= 128 ? 32 : (q.K >= 32 ? 8 : 1);
  Planned<float> pl = {};
  pl.split = {32, 1, 1};
  pl.plan.cluster = 1;
  if (lanes == 32 && !q.tA && q.tB && q.M % 4 == 0 && q.N % 4 == 0 && q.M * q.N >= 1024) {
    pl.plan.variant = kSmallNT;
    pl.plan.grid = dim3((unsigned)cgtb_ceil_div((q.M / 4) * (q.N / 4) * 32, 256), (unsigned)q.P);
  } else {
    pl.plan.variant = kSmall | lanes;
    pl.plan.grid = dim3((unsigned)cgtb_ceil_div(q.M * q.N * lanes, 256), (unsigned)q.P);
  }
  return run_product<float>(q, pl);
}
int product_variant(int dtype, int tA, int tB, long M, long N, long K) {
  if (dtype != cgtb_f4 || M <= 0 || N <= 0) return -1;
  return product_is_fma(tA, tB, 1, M, N, K) ? plan_product<float>(tA, tB, 1, M, N, K, true).plan.variant : -1;
}

}  // namespace cgtb

CGTB_API int cgtb_product_variant(int dtype, int tA, int tB, long M, long N, long K) {
  return cgtb::product_variant(dtype, tA, tB, M, N, K);
}
