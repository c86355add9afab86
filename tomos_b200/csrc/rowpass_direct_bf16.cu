// rowpass_direct_bf16.cu -- the direct row pass (rowpass_direct.cuh) over
// FP32_BF16 wh planes.
#include "rowpass_direct.cuh"

namespace tomos_b200 {

tomos_status launch_direct_bf16(bool acc64, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st) {
    return acc64 ? launch_direct_e<Elem::B16, true>(P, s, grid, st) : launch_direct_e<Elem::B16, false>(P, s, grid, st);
}

}  // namespace tomos_b200
