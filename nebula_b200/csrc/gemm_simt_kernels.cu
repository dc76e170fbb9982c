// The CUDA-core contraction for one pair of copy modes, NB_SIMT_A and NB_SIMT_B (CopyMode values the build gives).
#include "gemm_simt.cuh"

namespace nb {

template <>
const SimtVariant *simt_variants<NB_SIMT_A, NB_SIMT_B>() {
    static const SimtVariant v[SIMT_VARIANTS] = {
        simt_variant<NB_SIMT_A, NB_SIMT_B, 64, 128, 8, 8, 4>(), simt_variant<NB_SIMT_A, NB_SIMT_B, 64, 64, 8, 4, 4>(),
        simt_variant<NB_SIMT_A, NB_SIMT_B, 32, 64, 4, 4, 4>(), simt_variant<NB_SIMT_A, NB_SIMT_B, 16, 128, 4, 4, 4>()};
    return v;
}

}  // namespace nb
