// svpf_single_fast.cu -- single-filter tick through the fast sums.
#include "svpf_single.cuh"

namespace svpf {

cudaError_t launch_single_fast(const SingleArgs& a, int C, cudaStream_t s) {
    if (C < 2 || C > kMaxCluster || a.n < 1) return cudaErrorInvalidValue;
    const size_t smem = tick_smem_bytes_single_fast(a.n, C);
    if (smem > max_dyn_smem()) return cudaErrorInvalidValue;
    return launch_cluster(is_production_tick(a.cfg) ? single_fast_kernel<true> : single_fast_kernel<false>, a, C,
                          kWideThreads, smem, s);
}

}  // namespace svpf
