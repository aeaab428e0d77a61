// One matrix product, op(A) [M, K] . op(B) [K, N], and the kernels it can be given to.
#pragma once
#include "../../include/cgt_product.h"

namespace cgtb {

// A generated kernel that runs an elementwise chain on the elements of a product (codegen.product_source), compiled for
// one variant of the product kernels, with its operands. `part`, `nsplit`: only for the fold variants.
typedef int (*ChainLauncher)(const tile::Plan* plan, const void* args, const void* part, int nsplit, const void* const* in, const long* bk,
                             const long* bi, void* const* out, void* stream);
struct Chain {
  ChainLauncher launch;
  int variant;
  const void* const* in;
  const long *bk, *bi;
  void* const* out;
};

template <typename T>
struct Product {
  int tA, tB;
  long P, M, N, K;
  const T* A;
  long lda, strideA;
  const T* B;
  long ldb, strideB;
  T* C;
  long ldc, strideC;
  // output stages, at most one of them (P == 1): C = (addend + addend_bias) + (product + bias), or a chain that writes
  // its own results instead of C
  tile::Sums sums = {nullptr, nullptr, 0, nullptr};
  const Chain* chain = nullptr;
};

// The FMA kernels take a product below the size at which the tensor-core kernels' fixed cost (tensor-map fetch,
// tensor-memory allocation, a ring that a short K never fills: 10 - 15 us, 2 us more for the fold of a split K) is
// repaid: 39 M multiplications 8.4 and 15 us, 107 M (3200 x 512 x 65) 22 and 14 us. A batch of products of up to 2^25
// multiplications each stays with them whatever its length: 128 of 256^3 take 163 us here and 61 us on the tensor cores,
// but the three-fold TF32 split is off by 1.3e-6 (2-norm, against 64 bits) where plain float32 is off by 1.5e-7.
bool product_is_fma(int tA, int tB, long P, long M, long N, long K);
// 0 done, 1 error, -1: `chain` was compiled for another variant than this product needs. tiles_only: no small-product kernel
int product_fma(const Product<float>& q, bool tiles_only = false);
int product_fma(const Product<double>& q, bool tiles_only = false);
int product_small(const Product<float>& q);   // one warp per output; -1: not one of its shapes
int product_variant(int dtype, int tA, int tB, long M, long N, long K);

}  // namespace cgtb
