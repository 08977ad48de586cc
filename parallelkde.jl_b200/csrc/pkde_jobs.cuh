// Launches over the jobs of one or several estimations: blocks [block0[k], block0[k + 1]) are
// job k's.
#pragma once

#include "pkde_internal.cuh"

namespace pkde {

// The job of this block, copied into shared memory, and its first block.  Every thread calls.
template <class J>
__device__ __forceinline__ void find_job(const J *jobs, const unsigned *block0, int count, J &sj, unsigned &first) {
  __shared__ int s_job;
  if (threadIdx.x < 32) {
    int job = 0;
    for (;;) {  // block0 increases: the lanes at or below this block form a prefix
      const int k = job + 1 + (int)threadIdx.x;
      const bool le = k < count && __ldg(block0 + k) <= blockIdx.x;
      const int c = __popc(__ballot_sync(0xffffffffu, le));
      job += c;
      if (c < 32) break;
    }
    if (threadIdx.x == 0) s_job = job;
  }
  __syncthreads();
  const int job = s_job;
  const int *src = reinterpret_cast<const int *>(jobs + job);
  int *dst = reinterpret_cast<int *>(&sj);
  for (int i = threadIdx.x; i < (int)(sizeof(J) / sizeof(int)); i += blockDim.x) dst[i] = __ldg(src + i);
  first = __ldg(block0 + job);
  __syncthreads();
}

// Body::run(job, block) in T threads for each job.
template <class Body, class J, int T>
__global__ void __launch_bounds__(T) many_jobs_kernel(const J *jobs, const unsigned *block0, int count) {
  __shared__ J job;
  unsigned first;
  find_job(jobs, block0, count, job, first);
  Body::run(job, blockIdx.x - first);
}

}  // namespace pkde
