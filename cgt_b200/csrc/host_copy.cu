// Moving the arguments of a call into device memory and its results out of it.
//
// A call's small arrays are copied by ONE kernel at either end of its device work, which reads (writes) pinned host
// memory directly and is part of the captured graph; a call's large host arrays go through pinned memory in chunks of
// 256 KB, filled by up to four threads while the copy engine takes the chunks before (6.1 MB: 170 - 190 us, the driver's
// own staging of pageable memory 310 us; 1.6 MB: 75 and 91 us).
#include "copy_threads.h"
#include "host_copy.h"
#include "runtime.h"
#include <algorithm>
#include <cstring>
#include <mutex>

namespace cgtb {

namespace {
// blockIdx.y = job. Latency-bound (a read over PCIe takes about 1.5 us): two 16-byte loads per thread, issued together.
__global__ void __launch_bounds__(256) copy_jobs_kernel(const CopyJobs jobs) {
  const CopyJob j = jobs.job[blockIdx.y];
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
  const size_t both = (size_t)j.src | (size_t)j.dst;
  long done = 0;
  if ((both & 15) == 0) {
    const float4* s = (const float4*)j.src;
    float4* d = (float4*)j.dst;
    const long n = j.nbytes / 16;
    long i = t;
    for (; i + nt < n; i += 2 * nt) {
      const float4 a = s[i], b = s[i + nt];
      d[i] = a;
      d[i + nt] = b;
    }
    if (i < n) d[i] = s[i];
    done = n * 16;
  } else if ((both & 3) == 0) {
    const float* s = (const float*)j.src;
    float* d = (float*)j.dst;
    const long n = j.nbytes / 4;
    for (long i = t; i < n; i += nt) d[i] = s[i];
    done = n * 4;
  }
  for (long i = done + t; i < j.nbytes; i += nt) ((char*)j.dst)[i] = ((const char*)j.src)[i];
}
}  // namespace

const void* copy_jobs_function() { return (const void*)copy_jobs_kernel; }

void copy_jobs_launch_dims(const CopyJobs& jobs, unsigned* grid_x, unsigned* grid_y, unsigned* block) {
  long most = 1;
  for (int i = 0; i < jobs.n; ++i) most = std::max(most, jobs.job[i].nbytes);
  *grid_x = (unsigned)std::min<long>(cgtb_ceil_div(most, 256 * 32), (long)rt().sm_count * 8);
  *grid_y = (unsigned)jobs.n;
  *block = most <= 1024 ? 64 : 256;
}

int launch_copy_jobs(const CopyJobs& jobs) {
  if (jobs.n <= 0) return 0;
  unsigned gx, gy, block;
  copy_jobs_launch_dims(jobs, &gx, &gy, &block);
  CGTB_LAUNCH(copy_jobs_kernel, dim3(gx, gy), block, 0, jobs);
  CGTB_CHECK_LAUNCH("copy_jobs");
  return 0;
}

// ---------------------------------------------------------------- copies on the host
namespace {
CopyThreads g_copy_threads;

// Pinned memory that large arrays pass through, at most 32 MB; given back by cgtb_pool_trim.
struct Staging {
  static constexpr size_t kMost = 32 << 20;
  std::mutex mu;
  char* block = nullptr;
  size_t cap = 0, at = 0;
  cudaEvent_t emptied = nullptr;  // after the last copy out of `block`
  bool used = false;
};
Staging g_staging;
}  // namespace

void host_copy(void* dst, const void* src, size_t n) {
  // below a megabyte one thread is done before the helpers are awake
  if (n < ((size_t)1 << 20)) memcpy(dst, src, n);
  else g_copy_threads.copy((char*)dst, (const char*)src, n, false, [](size_t, size_t) {});
}

void stage_for_kernel(void* dst, const void* src, size_t n) {
  if (n < ((size_t)64 << 10)) memcpy(dst, src, n);
  else stream_to_pinned((char*)dst, (const char*)src, n);
}

int upload_pageable(void* dst, const void* src, size_t n) {
  if (n < ((size_t)1 << 20)) {  // the driver's own staging: 400 KB in 34 us; helpers would not be awake yet
    CGTB_CUDA_TRY(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, rt().stream));
    return 0;
  }
  Staging& s = g_staging;
  std::lock_guard<std::mutex> lk(s.mu);
  if (!s.emptied) CGTB_CUDA_TRY(cudaEventCreateWithFlags(&s.emptied, cudaEventDisableTiming));
  for (size_t from = 0; from < n; from += Staging::kMost) {
    const size_t part = std::min(Staging::kMost, n - from);
    if (s.used && cudaEventQuery(s.emptied) == cudaSuccess) s.at = 0;
    if (s.at + part > s.cap) {
      if (s.used) CGTB_CUDA_TRY(cudaEventSynchronize(s.emptied));
      s.at = 0;
      if (part > s.cap) {
        if (s.block) cudaFreeHost(s.block);
        s.block = nullptr;
        s.cap = 0;
        CGTB_CUDA_TRY(cudaHostAlloc((void**)&s.block, part, cudaHostAllocDefault));
        s.cap = part;
      }
    }
    char* stage = s.block + s.at;
    cudaError_t err = cudaSuccess;
    g_copy_threads.copy(stage, (const char*)src + from, part, true, [&](size_t a, size_t b) {
      if (err == cudaSuccess) err = cudaMemcpyAsync((char*)dst + from + a, stage + a, b - a, cudaMemcpyHostToDevice, rt().stream);
    });
    if (err != cudaSuccess) return fail("copy to the device failed: %s", cudaGetErrorString(err));
    CGTB_CUDA_TRY(cudaEventRecord(s.emptied, rt().stream));
    s.used = true;
    s.at += (part + 255) & ~(size_t)255;
  }
  return 0;
}

void trim_staging() {
  Staging& s = g_staging;
  std::lock_guard<std::mutex> lk(s.mu);
  if (s.used) cudaEventSynchronize(s.emptied);
  if (s.block) cudaFreeHost(s.block);
  s.block = nullptr;
  s.cap = s.at = 0;
}

}  // namespace cgtb

CGTB_API void cgtb_host_copy(void* dst, const void* src, long n) {
  if (n > 0) cgtb::host_copy(dst, src, (size_t)n);
}
