// Tensor-core GEMM over expanded weight codes, see gemm_tc.cuh (a compile unit per width, so that they build in parallel).
#include "gemm_tc.cuh"

namespace abq {
cudaError_t tc_launch_w0(const CUtensorMap &tw, const CUtensorMap &tx, const TcArgs &a, bool grouped, unsigned grid, size_t smem, cudaStream_t stream)
{
    return tc_launch_width<0>(tw, tx, a, grouped, grid, smem, stream);
}
} // namespace abq
