// FMA tiles with split K inside a thread-block cluster: the product kernel for everything below the size at which the
// tensor-core kernels' fixed cost is repaid, and for float64.
//
// What bounds such a product is not arithmetic but a chain of latencies: global loads, a barrier per K slice, a second
// launch where K is split. So the work is cut for length: a block of 256 threads owns one BT x BT tile of C, its four
// groups of 64 threads take different slices of K (each thread a BT/8 x BT/8 register tile, operands from shared memory
// by 16-byte reads whatever the storage order: nothing is transposed), the blocks of a cluster take different ranges of
// K, and the cluster folds the partial tiles through distributed shared memory in rank order. One launch, one fixed
// order of additions: reproducible. The next two slices of K are in flight (cp.async) while one is used.
//
// What happens to an element of the product is a template argument (`E`): the library stores it (Store), kernels that
// codegen.py generates run an elementwise chain on it.
//
// Storage orders: AK / BK true when the operand runs along K in memory. Shared tiles keep that order: [row][k] with a
// pitch of KT + 16 bytes or [k][row] with a pitch of BT.
#ifndef CGT_PRODUCT_H
#define CGT_PRODUCT_H
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "cgt_elwise.h"

namespace cgtb {
namespace tile {

// C = (addend + addend_bias) + (A.B + bias): row vectors bias, addend_bias [N], matrix addend [M, N]; any may be null.
struct Sums {
  const float* bias;
  const float* addend;
  long ldd;
  const float* addend_bias;
};

template <typename T>
struct Args {
  long M, N, K;
  const T *A, *B;
  long lda, ldb, stride_a, stride_b;
  T* C;                 // result, or the slabs of a K split over several clusters
  long ldc, stride_c;
  int tA, tB;
  int vec_a, vec_b;     // 16-byte loads are possible
  int tiles_n;
  int cluster, nsplit;  // K is cut into cluster * nsplit ranges of kchunk
  long kchunk;
  Sums sums;
};

template <typename T, int BT>
struct Shape {
  static constexpr int VW = 16 / (int)sizeof(T);
  static constexpr int KG = 64 / (int)sizeof(T);      // k of one group per slice
  static constexpr int KT = 4 * KG;                   // k of a slice
  static constexpr int PK = KT + VW;                  // pitch of a [row][k] tile
  static constexpr int TM = BT / 8;
  static constexpr int kStages = 3;
  static constexpr int kTile = BT * PK > KT * BT ? BT * PK : KT * BT;
  static constexpr int kStageBytes = 2 * kTile * (int)sizeof(T);
  static constexpr int kFoldBytes = 4 * BT * (BT + 1) * (int)sizeof(T);
  static constexpr int kSmem = kStages * kStageBytes > kFoldBytes ? kStages * kStageBytes : kFoldBytes;
};

template <int BYTES>
__device__ __forceinline__ void async_copy(unsigned s, const void* gmem, int valid) {
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(valid) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(s), "l"(gmem), "r"(valid), "n"(BYTES) : "memory");
}

// One operand's slices: rows [r0, r0 + BT) x k [k0, k0 + KT), zeros outside [0, R) x [.., kend). A thread copies the
// same chunks of every slice, so its addresses advance by a constant: address arithmetic would otherwise cost as many
// instructions as the multiplications.
template <typename T, int BT, bool ALONG_K>
struct Loader {
  using S = Shape<T, BT>;
  static constexpr int kPerLine = (ALONG_K ? S::KT : BT) / S::VW, kStep = 256 / kPerLine, kN = BT * S::KT / S::VW / 256;
  const T *p, *base;
  long line_step, slice_step;
  long k, kend;       // first k of the next slice (ALONG_K: of this thread's column of it)
  int rows_left;      // ALONG_K: R - first line of this thread; else: valid elements of its chunk (0 .. VW)
  bool vec;
  unsigned smem_at;

  __device__ __forceinline__ Loader(const T* g, long ld, long r0, long R, long kbegin, long kend_, bool vec_, int tid) {
    const int line = tid / kPerLine, at = (tid % kPerLine) * S::VW;
    base = g;
    kend = kend_;
    vec = vec_;
    if (ALONG_K) {
      p = g + (r0 + line) * ld + kbegin + at;
      line_step = kStep * ld;
      slice_step = S::KT;
      k = kbegin + at;
      const long left = R - (r0 + line);
      rows_left = left > BT ? BT : (int)left;
      smem_at = (unsigned)(line * S::PK + at) * (unsigned)sizeof(T);
    } else {
      p = g + (kbegin + line) * ld + r0 + at;
      line_step = kStep * ld;
      slice_step = S::KT * ld;
      k = kbegin + line;
      const long left = R - (r0 + at);
      rows_left = left > S::VW ? S::VW : (left < 0 ? 0 : (int)left);
      smem_at = (unsigned)(line * BT + at) * (unsigned)sizeof(T);
    }
  }
  __device__ __forceinline__ void next(unsigned tile) {
    const long kleft = kend - k;  // ALONG_K: valid elements of the chunk; else: valid lines
    const T* q = p;
    unsigned d = tile + smem_at;
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      int n;
      if (ALONG_K) n = i * kStep < rows_left ? (kleft >= S::VW ? S::VW : (kleft > 0 ? (int)kleft : 0)) : 0;
      else n = i * kStep < kleft ? rows_left : 0;
      if (vec) {
        async_copy<16>(d, n ? q : base, n * (int)sizeof(T));
      } else {
#pragma unroll
        for (int e = 0; e < S::VW; ++e) async_copy<(int)sizeof(T)>(d + e * (unsigned)sizeof(T), e < n ? q + e : base, e < n ? (int)sizeof(T) : 0);
      }
      q += line_step;
      d += (unsigned)(kStep * (ALONG_K ? S::PK : BT)) * (unsigned)sizeof(T);
    }
    p += slice_step;
    k += S::KT;
  }
};

template <typename T>
struct alignas(16) Vec {
  T v[16 / sizeof(T)];
};

// acc[i][j] += a[i] * b[j]. float with `pairs`: two products per instruction (fma.rn.f32x2 rounds each like fmaf); for
// a B tile stored along k its operands would first have to be moved together, which costs more than it saves.
template <int N, bool PAIRS>
__device__ __forceinline__ void outer_product(double (&acc)[N][N], const double (&a)[N], const double (&b)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
}
template <int N, bool PAIRS>
__device__ __forceinline__ void outer_product(float (&acc)[N][N], const float (&a)[N], const float (&b)[N]) {
  if (!PAIRS) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    return;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    unsigned long long aa;
    asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      unsigned long long bb, cc;
      asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b[j]), "f"(b[j + 1]));
      asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(acc[i][j]), "f"(acc[i][j + 1]));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][j]), "=f"(acc[i][j + 1]) : "l"(cc));
    }
  }
}

__device__ __forceinline__ double add_sums(const Sums&, long, long, double v) { return v; }
__device__ __forceinline__ float add_sums(const Sums& s, long m, long n, float v) {
  if (s.bias) v = __fadd_rn(v, s.bias[n]);
  if (s.addend) {
    float t = s.addend[m * s.ldd + n];
    if (s.addend_bias) t = __fadd_rn(t, s.addend_bias[n]);
    v = __fadd_rn(t, v);
  }
  return v;
}

// Default end of a product.
template <typename T>
struct Store {
  __device__ __forceinline__ void operator()(const Args<T>& a, int batch, long m, long n, T v) const {
    a.C[(long)batch * a.stride_c + m * a.ldc + n] = add_sums(a.sums, m, n, v);
  }
};

template <typename T, int BT, bool AK, bool BK, typename E>
__global__ void __launch_bounds__(256) gemm_tile_kernel(const __grid_constant__ Args<T> a, const __grid_constant__ E end_of) {
  using S = Shape<T, BT>;
  constexpr int VW = S::VW, KG = S::KG, KT = S::KT, PK = S::PK, TM = S::TM, NS = S::kStages;
  extern __shared__ __align__(16) unsigned char smem[];
  namespace cg = cooperative_groups;
  const int tid = threadIdx.x, group = tid >> 6, tx = tid & 7, ty = (tid >> 3) & 7;
  const int rank = (int)(blockIdx.z % a.cluster), z = (int)(blockIdx.z / a.cluster);
  const int split = z % a.nsplit, batch = z / a.nsplit;
  const long m0 = (long)(blockIdx.x / a.tiles_n) * BT, n0 = (long)(blockIdx.x % a.tiles_n) * BT;
  const T* A = a.A + (long)batch * a.stride_a;
  const T* B = a.B + (long)batch * a.stride_b;
  const long kbegin = ((long)split * a.cluster + rank) * a.kchunk;
  const long kend = kbegin + a.kchunk < a.K ? kbegin + a.kchunk : a.K;
  const int niter = kbegin < kend ? (int)((kend - kbegin + KT - 1) / KT) : 0;
  T* const tiles = (T*)smem;
  const unsigned tiles_at = (unsigned)__cvta_generic_to_shared(smem);
  Loader<T, BT, AK> la(A, a.lda, m0, a.M, kbegin, kend, a.vec_a != 0, tid);
  Loader<T, BT, BK> lb(B, a.ldb, n0, a.N, kbegin, kend, a.vec_b != 0, tid);
  auto load = [&](int it) {
    if (it < niter) {
      const unsigned s = tiles_at + (unsigned)((it % NS) * S::kStageBytes);
      la.next(s);
      lb.next(s + (unsigned)(S::kTile * sizeof(T)));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  T acc[TM][TM];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TM; ++j) acc[i][j] = T(0);
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) load(s);
  for (int it = 0; it < niter; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
    __syncthreads();
    load(it + NS - 1);
    const T* As = tiles + (it % NS) * (2 * S::kTile);
    const T* Bs = As + S::kTile;
#pragma unroll
    for (int kk = 0; kk < KG; kk += VW) {
      const int k = group * KG + kk;
      T av[VW][TM], bv[VW][TM];
      if (AK) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const Vec<T> t = *(const Vec<T>*)(As + (ty * TM + i) * PK + k);
#pragma unroll
          for (int q = 0; q < VW; ++q) av[q][i] = t.v[q];
        }
      } else {
#pragma unroll
        for (int q = 0; q < VW; ++q)
#pragma unroll
          for (int i = 0; i < TM; i += VW) {
            const Vec<T> t = *(const Vec<T>*)(As + (k + q) * BT + ty * TM + i);
#pragma unroll
            for (int e = 0; e < VW; ++e) av[q][i + e] = t.v[e];
          }
      }
      if (BK) {
#pragma unroll
        for (int j = 0; j < TM; ++j) {
          const Vec<T> t = *(const Vec<T>*)(Bs + (tx + 8 * j) * PK + k);
#pragma unroll
          for (int q = 0; q < VW; ++q) bv[q][j] = t.v[q];
        }
      } else {
#pragma unroll
        for (int q = 0; q < VW; ++q)
#pragma unroll
          for (int j = 0; j < TM; j += VW) {
            const Vec<T> t = *(const Vec<T>*)(Bs + (k + q) * BT + j * 8 + tx * VW);
#pragma unroll
            for (int e = 0; e < VW; ++e) bv[q][j + e] = t.v[e];
          }
      }
#pragma unroll
      for (int q = 0; q < VW; ++q) outer_product<TM, !BK>(acc, av[q], bv[q]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // fold the four groups: fold[g][m][n], pitch BT + 1
  T* fold = (T*)smem;
  constexpr int FP = BT + 1;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TM; ++j) {
      const int n = BK ? tx + 8 * j : (j / VW) * (8 * VW) + tx * VW + j % VW;
      fold[(group * BT + ty * TM + i) * FP + n] = acc[i][j];
    }
  __syncthreads();
  auto group_sum = [&](int e) {
    const int at = (e / BT) * FP + e % BT;
    return ((fold[at] + fold[BT * FP + at]) + fold[2 * BT * FP + at]) + fold[3 * BT * FP + at];
  };
  int first = tid, end = BT * BT;
  if (a.cluster > 1) {
    for (int e = tid; e < BT * BT; e += 256) fold[(e / BT) * FP + e % BT] = group_sum(e);
    cg::this_cluster().sync();
    first = rank * (BT * BT / a.cluster) + tid;
    end = (rank + 1) * (BT * BT / a.cluster);
  }
  auto total = [&](int e) {
    if (a.cluster == 1) return group_sum(e);
    const int at = (e / BT) * FP + e % BT;
    T part[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < a.cluster) part[s] = cg::this_cluster().map_shared_rank(fold, s)[at];
    T v = part[0];
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < a.cluster) v += part[s];
    return v;
  };
  for (int e = first; e < end; e += 256) {
    const long m = m0 + e / BT, n = n0 + e % BT;
    const T v = total(e);
    if (m >= a.M || n >= a.N) continue;
    if (a.nsplit > 1) a.C[((long)batch * a.nsplit + split) * a.M * a.N + m * a.N + n] = v;
    else end_of(a, batch, m, n, v);
  }
  if (a.cluster > 1) cg::this_cluster().sync();  // no block leaves while its partial tile may be read
}

// Few rows (M <= MR <= 8), B running along n: a lane owns a column, a warp every eighth k of its block's range, so that
// a warp reads 128 consecutive bytes of B per k and eight of them are in flight; the warps and then the blocks of the
// cluster are folded in order. Bound by the latency of those loads (1 x 256 x 784: 3 us; as 32 x 32 tiles 5.8 us).
template <typename T, int MR, typename E>
__global__ void __launch_bounds__(256) gemv_kernel(const __grid_constant__ Args<T> a, long sam, long sak, const __grid_constant__ E end_of) {
  namespace cg = cooperative_groups;
  __shared__ T fold[8][MR][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = (int)(blockIdx.z % a.cluster), batch = (int)(blockIdx.z / a.cluster);
  const long n = (long)blockIdx.x * 32 + lane;
  const T* A = a.A + (long)batch * a.stride_a;
  const T* B = a.B + (long)batch * a.stride_b + (n < a.N ? n : 0);
  const long kbegin = (long)rank * a.kchunk, kend = kbegin + a.kchunk < a.K ? kbegin + a.kchunk : a.K;
  T acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = T(0);
  for (long k0 = kbegin + warp; k0 < kend; k0 += 64) {
    T b[8], x[8][MR];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long k = k0 + 8 * u;
      const bool ok = k < kend;
      b[u] = ok ? B[k * a.ldb] : T(0);
#pragma unroll
      for (int m = 0; m < MR; ++m) x[u][m] = ok && m < a.M ? A[m * sam + k * sak] : T(0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int m = 0; m < MR; ++m) acc[m] = fma(x[u][m], b[u], acc[m]);
  }
#pragma unroll
  for (int m = 0; m < MR; ++m) fold[warp][m][lane] = acc[m];
  __syncthreads();
  const int m = warp;  // one warp per row from here on
  T v = T(0);
  if (m < MR) {
    v = fold[0][m][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) v += fold[w][m][lane];
  }
  if (a.cluster > 1) {
    __syncthreads();
    if (m < MR) fold[0][m][lane] = v;
    cg::this_cluster().sync();
    if (rank == 0 && m < MR) {
      T part[8];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < a.cluster) part[s] = cg::this_cluster().map_shared_rank(&fold[0][0][0], s)[m * 32 + lane];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < a.cluster) v += part[s];
    }
    cg::this_cluster().sync();
    if (rank != 0) return;
  }
  if (m < MR && m < a.M && n < a.N) end_of(a, batch, m, n, v);
}

// Adds the slabs of a K split over several clusters, in order, and finishes like the tile kernel.
template <typename T, typename E>
__global__ void __launch_bounds__(256) fold_kernel(const T* __restrict__ part, int nsplit, const __grid_constant__ Args<T> a, const __grid_constant__ E end_of) {
  const long total = a.M * a.N, e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const T* src = part + (long)blockIdx.y * nsplit * total + e;
  T v = src[0];
  int s = 1;
  for (; s + 8 <= nsplit; s += 8) {
    T t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = src[(long)(s + u) * total];
#pragma unroll
    for (int u = 0; u < 8; ++u) v += t[u];
  }
  for (; s < nsplit; ++s) v += src[(long)s * total];
  end_of(a, blockIdx.y, e / a.N, e % a.N, v);
}

// Products with few outputs and a short K (the classifier layer: 128 x 10 x 256 and its gradients):
// LANES consecutive threads share one output element, lane l taking k = l, l + LANES, ...; eight
// products' operands are loaded before the first multiply-add so that a thread has sixteen loads in
// flight (the kernel is bound by memory latency, not by bytes or flops). The lanes' sums are combined
// by a shuffle tree: a fixed order, so results are reproducible. A tiled kernel spends its time on
// pipeline fill and barriers for these shapes.
template <typename T, int LANES, typename E>
__global__ void small_kernel(const __grid_constant__ Args<T> g, const __grid_constant__ E end_of) {
  const long M = g.M, N = g.N, K = g.K;
  const long p = blockIdx.y;
  const long gthread = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long e = gthread / LANES;
  const int l = (int)(gthread % LANES);
  const bool live = e < M * N;
  const long ee = live ? e : 0;
  const long m = ee / N, n = ee - m * N;
  const T* a = g.A + p * g.stride_a + (g.tA ? m : m * g.lda);
  const T* b = g.B + p * g.stride_b + (g.tB ? n * g.ldb : n);
  const long sa = g.tA ? g.lda : 1, sb = g.tB ? 1 : g.ldb;
  T acc = T(0);
  for (long k0 = l; k0 < K; k0 += 8L * LANES) {
    T av[8], bv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long k = k0 + (long)u * LANES;
      const bool ok = live && k < K;
      av[u] = ok ? __ldg(a + k * sa) : T(0);
      bv[u] = ok ? __ldg(b + k * sb) : T(0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) acc = fma(av[u], bv[u], acc);
  }
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (live && l == 0) end_of(g, (int)p, m, n, acc);
}

// The same product when both operands run along K in memory (C = A . B^T, row-major A [M, K] and B [N, K]) and M, N are
// multiples of four: a warp owns a 4 x 4 block of outputs, so a row of A or B that it reads (one coalesced 128-byte
// load per 32 values of k) feeds four outputs instead of one: an eighth of the L2 traffic of one warp per output
// (64 x 128 x 512, the LSTM's hidden-state gradient: 33 MB of loads become 4 MB). Every output is still accumulated
// by lane l over k = l, l + 32, ... in ascending order and the lanes are folded by the same shuffle tree: the bits of
// small_kernel<32>.
template <typename T, typename E>
__global__ void __launch_bounds__(256) small_nt4_kernel(const __grid_constant__ Args<T> g, const __grid_constant__ E end_of) {
  const long M = g.M, N = g.N, K = g.K, lda = g.lda, ldb = g.ldb;
  const long p = blockIdx.y;
  const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int l = threadIdx.x & 31;
  const long nb = N / 4;
  if (w >= (M / 4) * nb) return;
  const long m0 = 4 * (w / nb), n0 = 4 * (w % nb);
  const T* a = g.A + p * g.stride_a + m0 * lda;
  const T* b = g.B + p * g.stride_b + n0 * ldb;
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
  constexpr int U = 8;   // 64 loads per lane in flight: the kernel is bound by the latency of its load rounds
  for (long k0 = l; k0 < K; k0 += 32 * U) {
    T av[U][4], bv[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long k = k0 + 32 * u;
      const bool ok = k < K;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[u][i] = ok ? __ldg(a + i * lda + k) : T(0);
        bv[u][i] = ok ? __ldg(b + i * ldb + k) : T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(av[u][i], bv[u][j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], d);
    }
  // every lane holds all sixteen sums: lanes 0 .. 15 finish one each
  T mine = T(0);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (l == 4 * i + j) mine = acc[i][j];
  if (l < 16) end_of(g, (int)p, m0 + l / 4, n0 + l % 4, mine);
}

// ------------------------------------------------------------------------------------------------
// Which kernel and how it is launched. `variant` names the kernel: a generated chain is compiled for one of them.
// ------------------------------------------------------------------------------------------------
enum : int { kSmall = 0x100, kSmallNT = 0x200, kRows = 0x300, kTiles = 0x400, kTilesFold = 0x800 };
struct Plan {
  int variant;    // kSmall | lanes, kSmallNT, kRows | MR, kTiles | (BT == 64) | AK << 1 | BK << 2, kTilesFold | the same
  dim3 grid;
  int cluster;
};

template <typename K, typename... A>
inline cudaError_t launch_cluster(K kernel, dim3 grid, int cluster, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = 256;
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = (unsigned)cluster;
  c.attrs = &attr;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, args...);
}

template <typename T, int VARIANT, typename E>
inline cudaError_t launch_tiles(const Plan& p, const Args<T>& a, const E& e, cudaStream_t stream) {
  constexpr int BT = (VARIANT & 1) ? 64 : 32;
  auto kernel = gemm_tile_kernel<T, BT, (VARIANT & 2) != 0, (VARIANT & 4) != 0, E>;
  constexpr int smem = Shape<T, BT>::kSmem;
  static const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (set != cudaSuccess) return set;
  return launch_cluster(kernel, p.grid, p.cluster, smem, stream, a, e);
}
// fold of the slabs at `part`, which a tile kernel left there
template <typename T, typename E>
inline cudaError_t launch_fold(const T* part, int nsplit, const Args<T>& a, long P, const E& e, cudaStream_t stream) {
  fold_kernel<T, E><<<dim3((unsigned)((a.M * a.N + 255) / 256), (unsigned)P), 256, 0, stream>>>(part, nsplit, a, e);
  return cudaPeekAtLastError();
}
template <typename T, int VARIANT, typename E>
inline cudaError_t launch_single(const Plan& p, const Args<T>& a, const E& e, cudaStream_t stream) {
  if constexpr ((VARIANT & 0xf00) == kTiles) return launch_tiles<T, VARIANT & 7>(p, a, e, stream);
  else if constexpr ((VARIANT & 0xf00) == kRows)
    return launch_cluster(gemv_kernel<T, VARIANT & 0xff, E>, p.grid, p.cluster, 0, stream, a, a.tA ? 1L : a.lda, a.tA ? a.lda : 1L, e);
  else if constexpr ((VARIANT & 0xf00) == kSmallNT) small_nt4_kernel<T, E><<<p.grid, 256, 0, stream>>>(a, e);
  else small_kernel<T, VARIANT & 0xff, E><<<p.grid, 256, 0, stream>>>(a, e);
  return cudaPeekAtLastError();
}

}  // namespace tile
}  // namespace cgtb
#endif
