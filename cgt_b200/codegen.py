"""Run-time code generation for elementwise Ops whose C expression is not one of the prebuilt ones.

Counterpart of the generated-kernel branch of ElwiseUnary.get_native_compile_info in the reference
(cgt/core.py:1216-1239): the expression string becomes a `__device__` function inside a vectorised
grid-stride kernel, compiled by nvcc for sm_100a into the hash-keyed library cache.
"""
import os

from . import core

_CUDA_TEMPLATE = r"""
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
__forceinline__ __device__ %(cdtype1)s scalar_$function(%(cdtype0)s x) { return %(cexpr)s; }
__global__ void ${function}_kernel(const long n, const %(cdtype0)s* __restrict__ in, %(cdtype1)s* __restrict__ out) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = scalar_$function(in[i]);
}
void launchker_$function(long n, const %(cdtype0)s* x, %(cdtype1)s* y, void* stream) {
  if (n <= 0) return;
  long blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  ${function}_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, x, y);
}
"""

_CPP_TEMPLATE = r"""
extern void launchker_${function}(long, const %(cdtype0)s*, %(cdtype1)s*, void*);
static inline %(cdtype1)s host_scalar_$function(%(cdtype0)s x) { return %(cexpr)s; }
CGT_EXPORT_C void $function(void* cldata, cgtArray** reads, cgtArray* write) {
    cgtArray* read = reads[0];
    long n = read->size();
    if (read->devtype() == cgtGPU) {
        launchker_$function(n, (const %(cdtype0)s*)read->data(), (%(cdtype1)s*)write->data(), cgt_current_stream());
    } else {
        cgt_check(n <= 64, "a tensor was placed on the host; this backend has no CPU implementation of tensor ops");
        for (long i = 0; i < n && n <= 64; ++i) write->at<%(cdtype1)s>(i) = host_scalar_$function(read->at<%(cdtype0)s>(i));
    }
}
"""


def unary_from_cexpr(op, input_types, devtype):
    out_dtype = op.typ_apply(input_types).dtype
    d = dict(cdtype0=core.np2c[input_types[0].dtype], cdtype1=core.np2c[out_dtype], cexpr=op.info.cexpr)
    return core.NativeCompileInfo(_CPP_TEMPLATE % d, includes=["math.h", "stdint.h"], link_flags="-lm",
                                  gpu_deref_mask=(True,), extra_srcs=[core.SrcFile("cuda", _CUDA_TEMPLATE % d)])


# ================================================================
# Fused elementwise chains
# ================================================================

_FUSED_HEAD = r"""
#include <cuda_runtime.h>
#include "cgt_elwise.h"
"""


def fused_source(op):
    """CUDA source of the kernel for one FusedElwise program. Every operation calls the scalar template
    the separate kernels use (float operands, literal opcode), values stay in registers, scalars are
    read once per thread. Compiled without multiply-add contraction: the separate kernels round every
    product before the next Op adds to it."""
    n_in = len(op.in_kinds)
    params, hoist, loads = [], [], []
    for (k, kind) in enumerate(op.in_kinds):
        if kind == 0:
            params.append("const float* __restrict__ in%d" % k)
            loads.append(("pack", "const Pack<float, V> p%d = load_pack<float, V>(in%d + i * V);" % (k, k), "p%d.v[v]" % k))
        elif kind == 1:
            params.append("const int8_t* __restrict__ in%d" % k)
            loads.append(("pack", "const Pack<int8_t, V> p%d = load_pack<int8_t, V>(in%d + i * V);" % (k, k), "(float)p%d.v[v]" % k))
        elif kind == 2:
            params.append("const float* __restrict__ in%d" % k)
            hoist.append("const float s%d = in%d[0];" % (k, k))
            loads.append(("none", "", "s%d" % k))
        elif kind == 3:
            params.append("const long* __restrict__ in%d" % k)
            hoist.append("const float s%d = (float)in%d[0];" % (k, k))
            loads.append(("none", "", "s%d" % k))
        elif kind == 7:
            # columns [bi, bi + W) of a matrix with rows of bk elements; W is a literal of this chain
            params.append("const float* __restrict__ in%d, const long bk%d, const long bi%d" % (k, k, k))
            W = op.static_shape[1]
            loads.append(("pack", "const I row%d = (i * V) / (I)%d;\n    const Pack<float, V> p%d = load_pack<float, V>(in%d + (size_t)row%d * bk%d + bi%d "
                          "+ ((i * V) - row%d * (I)%d));" % (k, W, k, k, k, k, k, k, W), "p%d.v[v]" % k))
        else:
            params.append("const float* __restrict__ in%d, const long bk%d, const long bi%d" % (k, k, k))
            # one value per pack when the run length is a multiple of V, else one index per element
            loads.append(("pack", "float b%d[V];\n    if ((I)bi%d %% V == 0) {\n      const float t = in%d[((i * V) / (I)bi%d) %% (I)bk%d];\n"
                          "#pragma unroll\n      for (int v = 0; v < V; ++v) b%d[v] = t;\n    } else {\n"
                          "#pragma unroll\n      for (int v = 0; v < V; ++v) b%d[v] = in%d[((i * V + v) / (I)bi%d) %% (I)bk%d];\n    }"
                          % (k, k, k, k, k, k, k, k, k, k), "b%d[v]" % k))
    outs = []
    for (q, dt) in enumerate(op.out_dtypes):
        ctype = "float" if dt == "f4" else "int8_t"
        params.append("%s* __restrict__ out%d" % (ctype, q))
        outs.append(ctype)
    lines = ["// I: index type (32-bit when the element count allows: the broadcast index needs a division)",
             "template <int V, typename I>", "__global__ void fused_kernel(const I n, %s) {" % ", ".join(params)]
    lines += ["  " + h for h in hoist]
    lines.append("  const I nv = n / V;")
    lines.append("  for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (I)gridDim.x * blockDim.x) {")
    for (_kind, stmt, _expr) in loads:
        if stmt:
            lines.append("    " + stmt)
    for (q, ctype) in enumerate(outs):
        lines.append("    Pack<%s, V> o%d;" % (ctype, q))
    lines.append("#pragma unroll")
    lines.append("    for (int v = 0; v < V; ++v) {")
    for (k, (_kind, _stmt, expr)) in enumerate(loads):
        lines.append("      const float r%d = %s;" % (k, expr))
    for (j, (arity, code, a, b)) in enumerate(op.program):
        if arity == 1:
            lines.append("      const float r%d = unary_apply<float, float>(%d, r%d);" % (n_in + j, code, a))
        else:
            lines.append("      const float r%d = binary_apply<float, float, float>(%d, r%d, r%d);" % (n_in + j, code, a, b))
    for (q, (reg, ctype)) in enumerate(zip(op.out_regs, outs)):
        lines.append("      o%d.v[v] = (%s)r%d;" % (q, ctype, reg))
    lines.append("    }")
    for (q, ctype) in enumerate(outs):
        lines.append("    store_pack<%s, V>(out%d + i * V, o%d);" % (ctype, q, q))
    lines += ["  }", "}"]
    args = []
    for (k, kind) in enumerate(op.in_kinds):
        ctype = {0: "float", 1: "int8_t", 2: "float", 3: "long", 4: "float", 7: "float"}[kind]
        args.append("(const %s*)in[%d]" % (ctype, k))
        if kind in (4, 7):
            args += ["bk[%d]" % k, "bi[%d]" % k]
    for (q, ctype) in enumerate(outs):
        args.append("(%s*)out[%d]" % (ctype, q))
    lines += [
        'extern "C" __attribute__((visibility("default"))) int cgtb_fused_launch(long n, const void* const* in, const long* bk,',
        "    const long* bi, void* const* out, int vectorised, void* stream, int sm_count) {",
        "  const long work = vectorised ? n / 4 : n;",
        "  long blocks = (work + 255) / 256;",
        "  if (blocks > (long)sm_count * 16) blocks = (long)sm_count * 16;",
        "  if (blocks < 1) blocks = 1;",
        "  const bool small = n < (1L << 31);",
        "  if (vectorised && small) fused_kernel<4, unsigned><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((unsigned)n, %s);" % ", ".join(args),
        "  else if (vectorised) fused_kernel<4, long><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, %s);" % ", ".join(args),
        "  else if (small) fused_kernel<1, unsigned><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((unsigned)n, %s);" % ", ".join(args),
        "  else fused_kernel<1, long><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, %s);" % ", ".join(args),
        "  return cudaPeekAtLastError() != cudaSuccess;",
        "}",
    ]
    return _FUSED_HEAD + "\n".join(lines) + "\n"


def rows_source(op):
    """CUDA source of the kernel for one FusedRows program: one warp per row, element c of the row in lane c % 32,
    slot c / 32; every operation calls the scalar template the separate kernels use; a row sum adds the lane's valid
    slots in order and then folds the lanes with xor shuffles (16, 8, 4, 2, 1), as the library's kernel does."""
    n_in = len(op.in_kinds)
    lines = ["template <int E>", "__global__ void __launch_bounds__(128) rows_kernel(const long R, const long C, const void* const* in_, void* const* out_) {"]
    params, args = [], []
    for (k, kind) in enumerate(op.in_kinds):
        ctype = "long" if kind in (3, 8) else "float"
        params.append("const %s* __restrict__ in%d" % (ctype, k))
        args.append("(const %s*)in[%d]" % (ctype, k))
    for q in range(len(op.out_regs)):
        params.append("float* __restrict__ out%d" % q)
        args.append("(float*)out[%d]" % q)
    lines = ["template <int E>",
             "__global__ void __launch_bounds__(128) rows_kernel(const long R, const long C, %s) {" % ", ".join(params),
             "  const int lane = threadIdx.x & 31;",
             "  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);",
             "  if (row >= R) return;"]
    for (k, kind) in enumerate(op.in_kinds):
        lines.append("  float r%d[E];" % k)
        if kind in (0, 6):
            base = "in%d + row * C" % k if kind == 0 else "in%d" % k
            lines += ["#pragma unroll", "  for (int e = 0; e < E; ++e) { const long c = lane + 32 * e; r%d[e] = c < C ? (%s)[c] : 0.0f; }" % (k, base)]
        elif kind == 8:
            lines += ["  { const long hot = in%d[row];" % k, "#pragma unroll",
                      "    for (int e = 0; e < E; ++e) r%d[e] = (lane + 32 * e == hot) ? 1.0f : 0.0f; }" % k]
        else:
            src = {5: "in%d[row]" % k, 2: "in%d[0]" % k, 3: "(float)in%d[0]" % k}[kind]
            lines += ["  { const float v = %s;" % src, "#pragma unroll", "    for (int e = 0; e < E; ++e) r%d[e] = v; }" % k]
    for (j, (arity, code, a, b)) in enumerate(op.program):
        d = n_in + j
        lines.append("  float r%d[E];" % d)
        if arity == 1:
            lines += ["#pragma unroll", "  for (int e = 0; e < E; ++e) r%d[e] = unary_apply<float, float>(%d, r%d[e]);" % (d, code, a)]
        elif arity == 2:
            lines += ["#pragma unroll", "  for (int e = 0; e < E; ++e) r%d[e] = binary_apply<float, float, float>(%d, r%d[e], r%d[e]);" % (d, code, a, b)]
        else:
            cond = "lane + 32 * e < C" if arity == 3 else "lane + 32 * e < C && r%d[e] != 0.0f" % b
            lines += ["  { float s = 0.0f;", "#pragma unroll", "    for (int e = 0; e < E; ++e) if (%s) s += r%d[e];" % (cond, a),
                      "#pragma unroll", "    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);",
                      "#pragma unroll", "    for (int e = 0; e < E; ++e) r%d[e] = s; }" % d]
    for (q, (reg, col)) in enumerate(zip(op.out_regs, op.out_cols)):
        if col:
            lines.append("  if (lane == 0) out%d[row] = r%d[0];" % (q, reg))
        else:
            lines += ["#pragma unroll", "  for (int e = 0; e < E; ++e) { const long c = lane + 32 * e; if (c < C) out%d[row * C + c] = r%d[e]; }" % (q, reg)]
    lines.append("}")
    call = "(R, C, %s)" % ", ".join(args)
    lines += [
        'extern "C" __attribute__((visibility("default"))) int cgtb_rows_launch(long R, long C, const void* const* in, void* const* out, void* stream) {',
        "  const unsigned blocks = (unsigned)((R + 3) / 4);",
        "  if (C <= 32) rows_kernel<1><<<blocks, 128, 0, (cudaStream_t)stream>>>%s;" % call,
        "  else if (C <= 64) rows_kernel<2><<<blocks, 128, 0, (cudaStream_t)stream>>>%s;" % call,
        "  else rows_kernel<4><<<blocks, 128, 0, (cudaStream_t)stream>>>%s;" % call,
        "  return cudaPeekAtLastError() != cudaSuccess;",
        "}",
    ]
    return _FUSED_HEAD + "\n".join(lines) + "\n"


def multi_source(op):
    """CUDA source of the kernel for one MultiFusedElwise: one program over up to 24 tensors of any sizes. Blocks are dealt
    out to the tensors by size (2048 elements each, two 16-byte groups per thread with all loads ahead of the arithmetic),
    so that neither a large tensor waits for few blocks nor a small one leaves blocks idle. Bound by HBM for large
    models: 12.6 M parameters of p - lr * g take 26 us, 86 us through the library's register machine."""
    fop = op.fused
    n_in, scalars = len(fop.in_kinds), [k for (k, kind) in enumerate(fop.in_kinds) if kind != 0]
    tensors = [k for (k, kind) in enumerate(fop.in_kinds) if kind == 0]
    reg = ["      const float r%d = %s;" % (k, "s%d" % k if k in scalars else "p%d[u].v[v]" % k) for k in range(n_in)]
    for (j, (arity, code, a, b)) in enumerate(fop.program):
        reg.append("      const float r%d = unary_apply<float, float>(%d, r%d);" % (n_in + j, code, a) if arity == 1 else
                   "      const float r%d = binary_apply<float, float, float>(%d, r%d, r%d);" % (n_in + j, code, a, b))
    out = fop.out_regs[0]
    lines = ["namespace {", "struct Job { const void* in[24][%d]; float* out[24]; long n[24]; unsigned first[25]; unsigned vec; int k; };" % n_in,
             "template <int V, int U>",
             "__device__ __forceinline__ void run(const Job& a, int t, long base) {",
             "  const long n = a.n[t] / V;"]
    for k in scalars:
        lines.append("  const float s%d = %s;" % (k, "((const float*)a.in[t][%d])[0]" % k if fop.in_kinds[k] == 2 else "(float)((const long*)a.in[t][%d])[0]" % k))
    for k in tensors:
        lines.append("  Pack<float, V> p%d[U];" % k)
    lines += ["#pragma unroll", "  for (int u = 0; u < U; ++u) {", "    const long i = base + u * 256 + threadIdx.x;", "    if (i < n) {"]
    lines += ["      p%d[u] = load_pack<float, V>((const float*)a.in[t][%d] + i * V);" % (k, k) for k in tensors]
    lines += ["    }", "  }", "#pragma unroll", "  for (int u = 0; u < U; ++u) {", "    const long i = base + u * 256 + threadIdx.x;", "    if (i >= n) continue;",
              "    Pack<float, V> o;", "#pragma unroll", "    for (int v = 0; v < V; ++v) {"] + reg
    lines += ["      o.v[v] = r%d;" % out, "    }", "    store_pack<float, V>(a.out[t] + i * V, o);", "  }", "}",
              "__global__ void __launch_bounds__(256) multi_kernel(const __grid_constant__ Job a) {",
              "  int t = 0;", "  while (t + 1 < a.k && blockIdx.x >= a.first[t + 1]) ++t;",
              "  const long b = blockIdx.x - a.first[t];",
              "  if ((a.vec >> t) & 1) {",
              "    run<4, 2>(a, t, b * 512);",
              "    if (b == 0 && threadIdx.x < (a.n[t] & 3)) {  // the last n % 4 elements",
              "      const long i = (a.n[t] & ~3L) + threadIdx.x;", "      Job one = a;", "      (void)one;"]
    # the tail is evaluated element by element with the same expressions
    tail = ["      const float r%d = %s;" % (k, "((const float*)a.in[t][%d])[%s]" % (k, "i" if k in tensors else "0") if fop.in_kinds[k] != 3 else
                                             "(float)((const long*)a.in[t][%d])[0]" % k) for k in range(n_in)]
    tail += [r for r in reg if not any(r.startswith("      const float r%d =" % k) for k in range(n_in))]
    lines[-2:] = []
    lines += tail + ["      a.out[t][i] = r%d;" % out, "    }", "  } else {", "    run<1, 8>(a, t, b * 2048);", "  }", "}", "}  // namespace",
              'extern "C" __attribute__((visibility("default"))) int cgtb_multi_launch(int k, const long* n, const void* const* in, void* const* out, void* stream) {',
              "  Job a;", "  a.k = k;", "  a.vec = 0;", "  unsigned blocks = 0;",
              "  for (int t = 0; t < k; ++t) {",
              "    bool vec = ((size_t)out[t] & 15) == 0;",
              "    for (int q = 0; q < %d; ++q) {" % n_in,
              "      a.in[t][q] = in[t * %d + q];" % n_in,
              "      if (%s) vec = vec && ((size_t)in[t * %d + q] & 15) == 0;" % (" || ".join("q == %d" % k for k in tensors) or "false", n_in),
              "    }",
              "    a.out[t] = (float*)out[t];", "    a.n[t] = n[t] > 0 ? n[t] : 0;", "    a.first[t] = blocks;", "    if (vec) a.vec |= 1u << t;",
              "    blocks += (unsigned)((a.n[t] + 2047) / 2048);", "  }", "  a.first[k] = blocks;", "  if (!blocks) return 0;",
              "  multi_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(a);", "  return cudaPeekAtLastError() != cudaSuccess;", "}"]
    return _FUSED_HEAD + "\n".join(lines) + "\n"


def multi_launcher(op):
    """Address of the generated launcher for a MultiFusedElwise, or None (the library's kernel runs it then)."""
    return _generated_launcher(multi_source(op), "multi_", "cgtb_multi_launch", "merged parameter updates")


def product_source(op):
    """CUDA source of the product kernel (include/cgt_product.h) whose output stage is the chain of one Mul22Chain: the
    chain's operations as in fused_source, on the element the product kernel has just finished."""
    chain, n_in = op.chain, len(op.chain.in_kinds)
    body = []
    for (k, kind) in enumerate(chain.in_kinds):
        if k == op.product:
            expr = "v"
        elif kind == 0:
            expr = "((const float*)in[%d])[i]" % k
        elif kind == 1:
            expr = "(float)((const int8_t*)in[%d])[i]" % k
        elif kind == 2:
            expr = "((const float*)in[%d])[0]" % k
        elif kind == 3:
            expr = "(float)((const long*)in[%d])[0]" % k
        elif kind == 7:
            expr = "((const float*)in[%d])[m * bk[%d] + bi[%d] + n]" % (k, k, k)
        else:
            expr = "((const float*)in[%d])[bi[%d] == 1 && bk[%d] == a.N ? n : (i / bi[%d]) %% bk[%d]]" % (k, k, k, k, k)
        body.append("    const float r%d = %s;" % (k, expr))
    for (j, (arity, code, x, y)) in enumerate(chain.program):
        if arity == 1:
            body.append("    const float r%d = unary_apply<float, float>(%d, r%d);" % (n_in + j, code, x))
        else:
            body.append("    const float r%d = binary_apply<float, float, float>(%d, r%d, r%d);" % (n_in + j, code, x, y))
    for (q, (reg, dt)) in enumerate(zip(chain.out_regs, chain.out_dtypes)):
        ctype = "float" if dt == "f4" else "int8_t"
        body.append("    ((%s*)out[%d])[i] = (%s)r%d;" % (ctype, q, ctype, reg))
    call = ("launch_fold<float>((const float*)part, nsplit, a, 1, c, (cudaStream_t)stream)" if op.variant & 0x800 else
            "launch_single<float, %d>(*plan, a, c, (cudaStream_t)stream)" % op.variant)
    n_out = len(chain.out_regs)
    lines = ['#include "cgt_product.h"', "using namespace cgtb::tile;",
             "namespace {  // internal linkage: the templates below are instantiated once per library, static variables included",
             "struct Chain {",
             "  const void* in[%d]; long bk[%d], bi[%d]; void* out[%d];" % (n_in, n_in, n_in, n_out),
             "  __device__ __forceinline__ void operator()(const Args<float>& a, int, long m, long n, float v) const {",
             "    const long i = m * a.N + n;"] + body + ["  }", "};", "}  // namespace"]
    lines += ['extern "C" __attribute__((visibility("default"))) int cgtb_product_launch(const Plan* plan, const void* args, const void* part, int nsplit,',
              "    const void* const* in, const long* bk, const long* bi, void* const* out, void* stream) {",
              "  const Args<float>& a = *(const Args<float>*)args;",
              "  Chain c;",
              "  for (int k = 0; k < %d; ++k) { c.in[k] = in[k]; c.bk[k] = bk[k]; c.bi[k] = bi[k]; }" % n_in,
              "  for (int q = 0; q < %d; ++q) c.out[q] = out[q];" % n_out,
              "  (void)plan; (void)part; (void)nsplit;",
              "  return %s != cudaSuccess;" % call, "}"]
    return "\n".join(lines) + "\n"


def product_launcher(op):
    """Address of the generated launcher for a Mul22Chain, or None: product and chain are separate launches then."""
    return _generated_launcher(product_source(op), "product_", "cgtb_product_launch", "a chain in a product's output stage")


def recurrence_plan(R, H, KA, N, n_act):
    """How a Recurrence is dealt out, or None when it does not fit. A cluster of C blocks owns RB rows through all steps;
    block c of it computes the N / H columns of UH of the H units. Its slice of W stays in registers for the whole launch:
    256 threads, one column each, KG of them sharing a column's K, KT values per thread. Chosen for the fewest
    multiply-adds per thread and step, RB * KT; of equals the smallest cluster, whose barrier is the cheapest."""
    NG, best = N // H, None
    for C in (1, 2, 4, 8):
        UH = -(-H // C)
        NC = NG * UH
        if NC > 256 or (C > 1 and UH * (C - 1) >= H):
            continue
        KG = 256 // NC
        KT = -(-(-(-KA // KG)) // 4) * 4
        KG = -(-KA // KT)
        RB = -(-R // (128 // C))
        shared = 4 * (2 * RB * KG * KT + KG * RB * NC)
        # 72 weights per thread leave registers for the sums and the chain. A thread per (row, unit) runs the chain, which ends
        # most plans: at 8 rows of 32 units a training step over 1024 examples takes 403 us, as separate launches 511. With
        # fewer units the limit of 8 rows ends them, which was not measured
        if KT > 72 or RB > 8 or RB * UH > 256 or shared > 46 * 1024:
            continue
        if best is None or RB * KT < best[0]:
            best = (RB * KT, dict(C=C, UH=UH, NC=NC, KG=KG, KT=KT, RB=RB, NG=NG))
    return best and best[1]


def recurrence_source(op):
    """CUDA source of the kernel for one Recurrence (plan: recurrence_plan). One step: every thread multiplies its KT
    weights (registers) with the rows' act (shared memory, broadcast reads), the K groups' partial sums meet in shared
    memory, one thread per (row, unit) adds them in order, runs the chain and writes its part of the next act into the
    shared memory of all blocks of the cluster; a cluster barrier ends the step, and what goes to global memory is written
    between a block's arrival there and its wait. The act is double-buffered, so one barrier
    per step is enough; the chain's other operands are loaded a step ahead.

    Bound by that serial chain, not by operations: the FMAs of a step (2 rows x 128 columns x 128 per block) take about
    300 cycles."""
    p = recurrence_plan(op.R, op.H, op.KA, op.N, len(op.act_spec))
    chain, n_in = op.chain, len(op.chain.in_kinds)
    states = sorted(op.state)
    per = int(op.bias) + len(op.external) + len(op.kept) + int(op.keep_act)
    ext0 = int(op.bias)
    regs, loads = [], []   # (type, name) of the operands that are loaded a step ahead
    if op.bias:
        for g in range(p["NG"]):
            regs.append("x%d" % g)
            loads.append("((const float*)q[0])[row * %d + %d + j]" % (op.N, g * op.H))
    for (pos, k) in enumerate(op.external):
        kind, src = chain.in_kinds[k], "q[%d]" % (ext0 + pos)
        regs.append("e%d" % k)
        loads.append({0: "((const float*)%s)[row * %d + j]" % (src, op.H), 2: "((const float*)%s)[0]" % src,
                      3: "(float)((const long*)%s)[0]" % src,
                      7: "((const float*)%s)[row * %d + %d + j]" % ((src,) + chain.views.get(k, (0, 0))[::-1])}[kind])
    L = ['namespace {',
         'constexpr int R = %d, H = %d, KA = %d, N = %d, C = %d, UH = %d, NC = %d, KG = %d, KT = %d, RB = %d, PER = %d;'
         % (op.R, op.H, op.KA, op.N, p["C"], p["UH"], p["NC"], p["KG"], p["KT"], p["RB"], per),
         'constexpr int KP = KG * KT, kPointers = %d;' % min(op.MAX_POINTERS, max(256, 1 << (per * op.steps - 1).bit_length())),
         'struct Job { const void* fixed[20]; int steps; const void* p[kPointers]; };',
         '// Warps come here from divergent code: they gather first, and every thread arrives for itself (no .aligned). Reached',
         '// without any condition in every step, the last one included: under one (s + 1 < steps, which the chain tests as well)',
         '// the two halves of a warp may take different ways to it. The results go to global memory between arrival and wait:',
         '// before the arrival, its release would wait for them.',
         '__device__ __forceinline__ void step_arrive() {',
         '  __syncwarp();',
         '  if (C > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");', '}',
         '__device__ __forceinline__ void step_wait() {',
         '  __syncwarp();',
         '  if (C > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");',
         '  else __syncthreads();', '}',
         '__device__ __forceinline__ void store_peer(float* own, int block, float v) {',
         '  if (C == 1) { *own = v; return; }',
         '  unsigned at;',
         '  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(own)), "r"(block));',
         '  asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(at), "f"(v) : "memory");', '}',
         '__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(256) recurrence_kernel(const __grid_constant__ Job a) {',
         '  __shared__ __align__(16) float act[2][RB][KP];',
         '  __shared__ float part[KG][RB][NC];',
         '  const int tid = threadIdx.x, u0 = (int)(blockIdx.x % C) * UH, row0 = (int)(blockIdx.x / C) * RB;',
         '  const int col = tid % NC, kg = tid / NC;',
         '  const bool multiplies = kg < KG;',
         '  const float* W = (const float*)a.fixed[1];',
         '  float w[KT];',
         '  {',
         '    const int unit = u0 + col % UH, n = (col / UH) * H + unit;',
         '#pragma unroll',
         '    for (int k = 0; k < KT; ++k) {',
         '      const int kk = kg * KT + k;',
         '      w[k] = multiplies && unit < H && kk < KA ? W[%s] : 0.0f;' % ("n * KA + kk" if op.tB else "kk * N + n"),
         '    }', '  }',
         '  for (int i = tid; i < RB * KP; i += 256) {',
         '    const int r = i / KP, k = i % KP;',
         '    act[0][r][k] = row0 + r < R && k < KA ? ((const float*)a.fixed[0])[(row0 + r) * KA + k] : 0.0f;',
         '    act[1][r][k] = 0.0f;',
         '  }',
         '  const int rr = tid / UH, u = tid % UH, j = u0 + u, row = row0 + rr;',
         '  const bool live = rr < RB && j < H && row < R;']
    if op.bias:
        for g in range(p["NG"]):
            L.append('  const float b%d = live ? ((const float*)a.fixed[2])[%d + j] : 0.0f, c%d = live ? ((const float*)a.fixed[3])[%d + j] : 0.0f;'
                     % (g, g * op.H, g, g * op.H))
    for (pos, k) in enumerate(states):
        L.append('  float t%d = live ? ((const float*)a.fixed[%d])[row * H + j] : 0.0f;' % (k, 2 + 2 * op.bias + pos))
    L += ['  float %s;' % ", ".join("%s = 0.0f, next_%s = 0.0f" % (r, r) for r in regs)] if regs else []
    fetch = ['      next_%s = %s;' % (r, ld) for (r, ld) in zip(regs, loads)]
    L += ['  if (live) {', '    const void* const* q = a.p;', '    (void)q;'] + fetch + ['  }',
          '  step_arrive();', '  step_wait();',
          '  for (int s = 0; s < a.steps; ++s) {',
          '    const void* const* now = a.p + s * PER;', '    (void)now;']
    L += ['    %s = next_%s;' % (r, r) for r in regs]
    L += ['    if (live) {  // a step ahead; the last one again at the end', '      const void* const* q = a.p + (s + 1 < a.steps ? s + 1 : s) * PER;',
          '      (void)q;'] + fetch + ['    }',
          '    if (multiplies) {',
          '      float sum[RB];',
          '#pragma unroll',
          '      for (int r = 0; r < RB; ++r) sum[r] = 0.0f;',
          '      const float* x = &act[s & 1][0][kg * KT];',
          '#pragma unroll',
          '      for (int k = 0; k < KT; k += 4) {',
          '#pragma unroll',
          '        for (int r = 0; r < RB; ++r) {',
          '          const float4 v = *reinterpret_cast<const float4*>(x + r * KP + k);',
          '          sum[r] = fmaf(v.x, w[k], sum[r]);', '          sum[r] = fmaf(v.y, w[k + 1], sum[r]);',
          '          sum[r] = fmaf(v.z, w[k + 2], sum[r]);', '          sum[r] = fmaf(v.w, w[k + 3], sum[r]);',
          '        }', '      }',
          '#pragma unroll',
          '      for (int r = 0; r < RB; ++r) part[kg][r][col] = sum[r];',
          '    }',
          '    __syncthreads();']
    stored = sorted(set(op.kept) | {q for (q, _off) in op.act_spec} | {op.state[k] for k in states})
    L += ['    float %s;' % ", ".join("o%d = 0.0f" % q for q in stored), '    if (live) {']
    for g in range(p["NG"]):
        L += ['      float z%d = part[0][rr][%d + u];' % (g, g * p["UH"]), '#pragma unroll',
              '      for (int k = 1; k < KG; ++k) z%d += part[k][rr][%d + u];' % (g, g * p["UH"])]
        if op.bias:
            L.append('      z%d = (x%d + c%d) + (z%d + b%d);' % (g, g, g, g, g))
    for k in range(n_in):
        src = "z%d" % (op.z_inputs[k] // op.H) if k in op.z_inputs else "t%d" % k if k in op.state else "e%d" % k
        L.append('      const float r%d = %s;' % (k, src))
    for (i, (arity, code, x, y)) in enumerate(chain.program):
        L.append('      const float r%d = %s;' % (n_in + i, "unary_apply<float, float>(%d, r%d)" % (code, x) if arity == 1 else
                                                  "binary_apply<float, float, float>(%d, r%d, r%d)" % (code, x, y)))
    L += ['      o%d = r%d;' % (q, chain.out_regs[q]) for q in stored]
    L += ['      t%d = o%d;' % (k, op.state[k]) for k in states]
    L += ['      float* dst = &act[(s + 1) & 1][rr][j];',
          '#pragma unroll', '      for (int c = 0; c < C; ++c) {']
    L += ['        store_peer(dst + %d, c, o%d);' % (off, q) for (q, off) in op.act_spec]
    L += ['      }', '    }', '    step_arrive();', '    if (live) {']
    at = ext0 + len(op.external)
    for (pos, q) in enumerate(op.kept):
        L.append('      ((float*)now[%d])[row * H + j] = o%d;' % (at + pos, q))
    if op.keep_act:
        for (q, off) in op.act_spec:
            L.append('      ((float*)now[%d])[row * KA + %d + j] = o%d;' % (at + len(op.kept), off, q))
    L += ['    }', '    step_wait();',
          '  }', '}', '}  // namespace',
          'extern "C" __attribute__((visibility("default"))) int cgtb_recurrence_launch(int steps, const void* const* fixed,',
          '    const void* const* per_step, void* stream) {',
          '  if (steps < 1 || steps * PER > kPointers) return 1;',
          '  Job a;',
          '  for (int k = 0; k < %d; ++k) a.fixed[k] = fixed[k];' % (2 + 2 * op.bias + len(states)),
          '  a.steps = steps;',
          '  for (int k = 0; k < steps * PER; ++k) a.p[k] = per_step[k];',
          '  recurrence_kernel<<<C * ((R + RB - 1) / RB), 256, 0, (cudaStream_t)stream>>>(a);',
          '  return cudaPeekAtLastError() != cudaSuccess;', '}']
    return _FUSED_HEAD + "\n".join(L) + "\n"


def recurrence_launcher(op):
    """Address of the generated launcher for a Recurrence, or None: its steps stay separate launches then."""
    return _generated_launcher(recurrence_source(op), "recurrence_", "cgtb_recurrence_launch", "the steps of a recurrent network")


_fused_libs = {}


def rows_launcher(op):
    """Address of the generated launcher for a FusedRows program, or None (the library's kernel runs it then)."""
    return _generated_launcher(rows_source(op), "rows_", "cgtb_rows_launch", "a fused row chain")



def fused_launcher(op):
    """Address of the generated launcher for this program (compiled into the hash-keyed cache on first
    use), or None when generation is switched off or the compiler is not available: the library's
    register-machine kernel then runs the program."""
    return _generated_launcher(fused_source(op), "fused_", "cgtb_fused_launch", "a fused elementwise chain")


def generate_all(ops):
    """Generate and compile the kernels of these Ops that are not in the cache yet, several compilers at a time; the
    number of Ops that have a generated kernel."""
    import concurrent.futures
    makers = {core.FusedElwise: fused_launcher, core.MultiFusedElwise: multi_launcher, core.FusedRows: rows_launcher, core.Mul22Chain: product_launcher,
              core.Recurrence: recurrence_launcher}
    sources = {core.FusedElwise: fused_source, core.MultiFusedElwise: multi_source, core.FusedRows: rows_source, core.Mul22Chain: product_source,
               core.Recurrence: recurrence_source}
    todo, n = {}, 0
    for op in ops:
        if type(op) in makers:
            todo.setdefault((type(op), sources[type(op)](op)), []).append(op)
    if not core.get_config().get("jit_fused_elementwise", True):
        return 0
    (config, floatX) = (core.get_config(), core.float_dtype())

    def make(op):
        with core.options_of_thread(config, floatX):
            return makers[type(op)](op)
    with concurrent.futures.ThreadPoolExecutor(8) as pool:
        for (same, addr) in zip(todo.values(), pool.map(lambda same: make(same[0]), todo.values())):
            n += len(same) if addr else 0
    return n


_product_header_text = None


def _product_header():
    """The product kernels are compiled into the generated library: it is as old as this text."""
    global _product_header_text
    if _product_header_text is None:
        import os.path as osp
        from . import runtime
        with open(osp.join(runtime.INCLUDE_DIR, "cgt_product.h")) as fh:
            _product_header_text = fh.read()
    return _product_header_text


def _generated_launcher(src, tag, symbol, what):
    import ctypes
    import os.path as osp
    import threading
    from . import compilation, utils
    if not core.get_config().get("jit_fused_elementwise", True):
        return None
    info = compilation.get_compile_info()
    prefix = tag + utils.hash_seq1(src, "fmad=false", str(compilation.CPP_ABI_VERSION), *([_product_header()] if tag == "product_" else []))
    if prefix in _fused_libs:
        return _fused_libs[prefix][1]
    libpath = osp.join(info["CACHE_ROOT"], prefix + ".so")
    try:
        if not osp.exists(libpath):
            # files of this thread's own until they are complete: other ranks and threads may want the same kernel
            (srcpath, mine) = (osp.join(info["CACHE_ROOT"], prefix + ".cu"), "%d.%d" % (os.getpid(), threading.get_ident()))
            with open("%s.%s.cu" % (srcpath, mine), "w") as fh:
                fh.write(src)
            compilation._call("nvcc %s.%s.cu -o %s.%s.tmp -shared -gencode arch=compute_100a,code=sm_100a -lineinfo -O3 -std=c++17 "
                              "-fmad=false -Xcompiler -fPIC %s -L/usr/local/cuda/lib64 -lcudart"
                              % (srcpath, mine, libpath, mine, info["INCLUDES"]))
            os.replace("%s.%s.cu" % (srcpath, mine), srcpath)
            os.replace("%s.%s.tmp" % (libpath, mine), libpath)
        lib = ctypes.CDLL(libpath)
        addr = ctypes.cast(getattr(lib, symbol), ctypes.c_void_p).value
    except (RuntimeError, OSError) as err:
        import sys
        sys.stderr.write("cgt_b200: no generated kernel for %s (%s); using the built-in one\n" % (what, str(err).splitlines()[0]))
        _fused_libs[prefix] = (None, None)
        return None
    _fused_libs[prefix] = (lib, addr)
    return addr
