// qz_pipeline_o5.cu -- the pipelined kernel for Adams-Bashforth order 5 (qz_pipeline_kernels.cuh).
#include "qz_pipeline_kernels.cuh"

namespace qzb {

template <>
cudaError_t pipeline_launch_ord<5>(const PipeArgs& P, int grid, size_t smem, cudaStream_t s) {
    return launch_o<5>(P, grid, smem, s);
}

template <>
int pipeline_occupancy_ord<5>(const PipeArgs& P, size_t smem, int nsm) {
    return occupancy_o<5>(P, smem, nsm);
}

}  // namespace qzb
