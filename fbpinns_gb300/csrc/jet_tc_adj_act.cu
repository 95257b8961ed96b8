// Tensor-core adjoint for the other activations: SIREN, AdaptiveFCN and
// AdaptiveSIREN.
#include "jet_tc_adj_launch.cuh"

namespace fbp {
int tc_adj_group_act(int mode, const fbp_net* net, const float* x, const fbp_pairs* pr, const float* slot_out,
                     float* grad_part, int32_t* status, int grid, cudaStream_t st) {
    FBP_TC_ADJ_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_SIN)
    FBP_TC_ADJ_TRY(2, 16, 1, FBP_ACT_SIN)
    FBP_TC_ADJ_TRY(1, 32, 1, FBP_ACT_SIN)
    FBP_TC_ADJ_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_ADAPTIVE_TANH)
    FBP_TC_ADJ_TRY(2, 16, 1, FBP_ACT_ADAPTIVE_TANH)
    FBP_TC_ADJ_TRY(1, 32, 1, FBP_ACT_ADAPTIVE_TANH)
    FBP_TC_ADJ_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_ADAPTIVE_SIN)
    FBP_TC_ADJ_TRY(2, 16, 1, FBP_ACT_ADAPTIVE_SIN)
    FBP_TC_ADJ_TRY(1, 32, 1, FBP_ACT_ADAPTIVE_SIN)
    return 1;
}
}  // namespace fbp
