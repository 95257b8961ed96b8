// Tensor-core forward for tanh networks with two 16- or 32-wide hidden layers.
#include <algorithm>
#include <atomic>

#include "jet_tc_fwd.cuh"

namespace fbp {
int tc_group_tanh(int mode, const fbp_net* net, const float* x, const fbp_pairs* pr, float* pair_out, int32_t* status,
                int grid, cudaStream_t st) {
#define FBP_TM_TRY(XD, H, D2)                                                                 \
    {                                                                                         \
        int r_ = tm_try<XD, H, D2>(mode, *net, x, *pr, pair_out, status, grid, st);           \
        if (r_ != 1) return r_;                                                               \
    }
    FBP_TM_TRY(2, 16, 3 | FBP_D2_LAPLACIAN)
    FBP_TM_TRY(2, 16, 3)
    FBP_TM_TRY(2, 16, 1)
    FBP_TM_TRY(2, 16, 0)
    FBP_TM_TRY(1, 32, 1)
    FBP_TM_TRY(1, 32, 0)
    FBP_TM_TRY(2, 32, 3 | FBP_D2_LAPLACIAN)
    FBP_TM_TRY(2, 32, 3)
    FBP_TM_TRY(2, 32, 0)
    FBP_TM_TRY(3, 32, 7 | FBP_D2_GROUP(3))
    FBP_TM_TRY(3, 32, 7)
    FBP_TM_TRY(3, 32, 0)
#undef FBP_TM_TRY
    return 1;
}
}  // namespace fbp
