// Instantiates the kernel of 256 x 512 tiles for one operand kind; included once by each tc_wide_*.cu so that the kinds compile
// in parallel.
#include "tc_wide.cuh"

namespace kb {

namespace tc {

template <>
cudaError_t launch_wide_kind<KB_TC_KIND>(const TcPlan &plan, const void *tmap_out, const WideParams &p, cudaStream_t stream)
{
    return launch_wide_one<KB_TC_KIND>(plan, tmap_out, p, stream);
}

}  // namespace tc

}  // namespace kb
