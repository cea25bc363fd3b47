// Generator expansion of one statement (src/commitment/sis.rs:212-245).
#include <cuda_runtime.h>

#include "dm_blake3.cuh"
#include "dm_jobs.cuh"
#include "dm_kernels.cuh"

namespace dm {

// The generator expansion of one statement through the multi-job kernel the
// prover uses (gen_jobs_kernel, k_jobs.cu), as a single job.
cudaError_t launch_gen_generators(const uint8_t g_seed[32], uint64_t N, uint32_t log_n, uint4* d_g,
                                  cudaStream_t st, bool beside) {
    GenJob job{};
    for (int i = 0; i < 8; ++i) job.key[i] = b3_load_le32(g_seed + 4 * i);
    job.dst = d_g;
    job.total = N * kRank << log_n;
    job.log_n = log_n;
    if (job.total == 0) return cudaSuccess;
    return launch_gen_jobs(&job, 1, st, beside);
}

}  // namespace dm
