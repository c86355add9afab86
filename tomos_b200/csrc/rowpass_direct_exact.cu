// rowpass_direct_exact.cu -- the direct row pass (rowpass_direct.cuh) over
// both planes of packed storage (always FP64 sums).
#include "rowpass_direct.cuh"

namespace tomos_b200 {

tomos_status launch_direct_exact(Elem e, const DirectParams& P, const DirectShape& s, int grid, cudaStream_t st) {
    switch (e) {
        case Elem::A16: return launch_direct_e<Elem::A16, true>(P, s, grid, st);
        case Elem::AB16: return launch_direct_e<Elem::AB16, true>(P, s, grid, st);
        default: return launch_direct_e<Elem::AB16R, true>(P, s, grid, st);
    }
}

}  // namespace tomos_b200
