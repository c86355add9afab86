// rowpass_direct_f32.cu -- the direct row pass (rowpass_direct.cuh) over FP32.
#include "rowpass_direct.cuh"

namespace tomos_b200 {

tomos_status launch_direct_f32(bool acc64, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st) {
    return acc64 ? launch_direct_e<Elem::F32, true>(P, s, grid, st) : launch_direct_e<Elem::F32, false>(P, s, grid, st);
}

}  // namespace tomos_b200
