// Moving the arguments of a call into device memory and its results out of it (host_copy.cu).
#pragma once
#include <cstddef>

namespace cgtb {

// One contiguous copy between any two addresses the GPU can reach: device memory or pinned host memory.
struct CopyJob {
  const void* src;
  void* dst;
  long nbytes;
};
constexpr int kMaxCopyJobs = 32;
struct CopyJobs {
  CopyJob job[kMaxCopyJobs];
  int n;
};

// Host arrays up to this size are moved by copy_jobs_kernel through pinned memory, larger ones by the copy engine.
// Inside a graph of six small kernels a copy of 128 KB in and 512 bytes out took 20.1 us with the kernel at both ends
// and 35.8 us with memcpy nodes (3 KB: 14.9 and 26.5 us): a change between the compute and the copy engine costs about
// five microseconds each way. From a quarter of a megabyte on the copy engine's bandwidth repays that.
constexpr long kKernelCopyBytes = 256 << 10;

int launch_copy_jobs(const CopyJobs& jobs);   // one kernel on the runtime stream
const void* copy_jobs_function();             // the kernel, to find its node in a captured graph
void copy_jobs_launch_dims(const CopyJobs& jobs, unsigned* grid_x, unsigned* grid_y, unsigned* block);

// memcpy by several threads when the block is large
void host_copy(void* dst, const void* src, size_t nbytes);
// pageable host memory -> device on the runtime stream; `src` may be reused on return
int upload_pageable(void* dst_device, const void* src, size_t nbytes);
// fills a pinned block that copy_jobs_kernel reads
void stage_for_kernel(void* dst, const void* src, size_t nbytes);
void trim_staging();
// whether `p` is the start of a pinned block of the runtime's own pools
bool host_block_is_pinned(const void* p);

}  // namespace cgtb
