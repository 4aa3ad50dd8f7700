// Instantiates the tensor-core kernels of one operand kind; included once by each tc_inst_*.cu so that the kinds compile in
// parallel.
#include "tc_kernel.cuh"

namespace kb {

namespace tc {

template <>
cudaError_t launch_kind<KB_TC_KIND>(const TcPlan &plan, const TcParams &p, cudaStream_t stream)
{
    if (plan.pair) {
        return launch_one<KB_TC_KIND, 256, true>(plan, p, stream);
    }
    return plan.block_n > 128 ? launch_one<KB_TC_KIND, 256, false>(plan, p, stream)
                               : launch_one<KB_TC_KIND, 128, false>(plan, p, stream);
}

template <>
int pair_clusters_kind<KB_TC_KIND>(size_t smem_bytes)
{
    return max_pair_clusters<KB_TC_KIND>(smem_bytes);
}

}  // namespace tc

}  // namespace kb
