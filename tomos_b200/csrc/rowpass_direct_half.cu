// rowpass_direct_half.cu -- the direct row pass (rowpass_direct.cuh) over
// fp16 storage and FP32_16 wh planes.
#include "rowpass_direct.cuh"

namespace tomos_b200 {

tomos_status launch_direct_half(Elem e, bool acc64, const DirectParams& P, const DirectShape& s, int grid,
                                cudaStream_t st) {
    if (e == Elem::F16)
        return acc64 ? launch_direct_e<Elem::F16, true>(P, s, grid, st)
                     : launch_direct_e<Elem::F16, false>(P, s, grid, st);
    return acc64 ? launch_direct_e<Elem::H16, true>(P, s, grid, st) : launch_direct_e<Elem::H16, false>(P, s, grid, st);
}

}  // namespace tomos_b200
