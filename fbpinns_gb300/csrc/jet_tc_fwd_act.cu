// Tensor-core forward for the other activations of 2-16-16-1 networks: SIREN,
// AdaptiveFCN, AdaptiveSIREN and FourierFCN with 8 features.  (1-32-32-1 networks
// with them keep the FMA forward: the 1D oscillator's few hundred pairs are one
// tile per network, where both take the same time.)
#include "jet_tc_fwd.cuh"

namespace fbp {
int tc_fwd_group_act(int mode, const fbp_net* net, const float* x, const fbp_pairs* pr, float* pair_out,
                     int32_t* status, int grid, cudaStream_t st) {
    FBP_TM_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_SIN)
    FBP_TM_TRY(2, 16, 1, FBP_ACT_SIN)
    FBP_TM_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_ADAPTIVE_TANH)
    FBP_TM_TRY(2, 16, 1, FBP_ACT_ADAPTIVE_TANH)
    FBP_TM_TRY(2, 16, 3 | FBP_D2_LAPLACIAN, FBP_ACT_ADAPTIVE_SIN)
    FBP_TM_TRY(2, 16, 1, FBP_ACT_ADAPTIVE_SIN)
    FBP_TM_TRY(2, 16, 1, FBP_ACT_FOURIER)
    return 1;
}
}  // namespace fbp
