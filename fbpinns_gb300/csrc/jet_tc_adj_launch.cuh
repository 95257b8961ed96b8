// Launch wrapper of the tensor-core adjoint for one compiled shape; included by
// the translation units that instantiate them.
#pragma once

#include <algorithm>
#include <mutex>

#include "jet_tc_adj.cuh"

namespace fbp {

template <int XD, int H, int D2, int ACT>
int launch_adjoint_tc(const fbp_net& net, const float* x, const fbp_pairs& pr, const float* slot_out,
                      float* grad_part, int32_t* status, int grid, cudaStream_t st) {
    using C = TcCfg<Cfg<XD, H, H, D2, ACT>>;
    constexpr int threads = TcAdj<C>::T;
    FBP_REQUIRE(net.nparam == C::P, FBP_ERR_INVALID, "adjoint_tc: nparam %d != %d for this shape", net.nparam, C::P);
    struct Launch {
        int res;     // resident CTAs per SM
        size_t shm;  // dynamic shared memory per CTA
    };
    static Launch launch_dev[FBP_MAX_DEVICES] = {};
    static std::mutex launch_mu;  // the first launch per device sets both fields; others read a copy
    const int dev = current_device();
    constexpr int cols = TcAdj<C>::COLS;
    Launch L;
    {
        std::lock_guard<std::mutex> lock(launch_mu);
        Launch& cached = launch_dev[dev];
        if (!cached.res) {
            size_t shm = sizeof(TcAdjSmem<C>);
            FBP_CUDA_CHECK(cudaFuncSetAttribute(adjoint_pairs_tc_kernel<C>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
            cudaFuncAttributes fa;
            FBP_CUDA_CHECK(cudaFuncGetAttributes(&fa, adjoint_pairs_tc_kernel<C>));
            int smem_sm = 0, regs_sm = 0, thr_sm = 0;
            FBP_CUDA_CHECK(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
            FBP_CUDA_CHECK(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev));
            FBP_CUDA_CHECK(cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev));
            const int per_cta_smem = (int)(shm + fa.sharedSizeBytes) + 1024;  // + the runtime's 1 KiB per CTA
            const int per_cta_regs = ((fa.numRegs + 7) / 8 * 8) * threads;
            int res = std::min(std::min(smem_sm / per_cta_smem, regs_sm / std::max(per_cta_regs, 1)), thr_sm / threads);
            FBP_REQUIRE(res >= 1, FBP_ERR_UNSUPPORTED, "adjoint_tc: kernel does not fit on an SM");
            // a CTA beyond 512 / COLS TMEM columns per SM would block in tcgen05.alloc:
            // pad the shared-memory request until no more than that many fit
            const int max_res = 512 / cols;
            if (res > max_res) {
                const int pad_cta = smem_sm / max_res;
                shm = (size_t)(pad_cta - (int)fa.sharedSizeBytes - 1024);
                FBP_CUDA_CHECK(cudaFuncSetAttribute(adjoint_pairs_tc_kernel<C>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
                res = max_res;
            }
            cached.shm = shm;
            cached.res = res;
        }
        L = cached;
    }
    FBP_REQUIRE(L.res * cols <= 512, FBP_ERR_UNSUPPORTED, "adjoint_tc: %d CTAs/SM x %d TMEM columns > 512", L.res,
                cols);
    if (grid <= 0) grid = (int)std::min<int64_t>(L.res * sm_count(), std::max<int64_t>(pr.items_cap, 1));
    if (pr.item_ctr) FBP_CUDA_CHECK(cudaMemsetAsync(pr.item_ctr, 0, sizeof(int32_t), st));
    FBP_CUDA_CHECK(launch_after(adjoint_pairs_tc_kernel<C>, grid, threads, L.shm, st, net, x, pr, slot_out, grad_part,
                                status));
    return FBP_OK;
}

template <int XD, int H, int D2, int ACT>
int tc_adj_try(int mode, const fbp_net& net, const float* x, const fbp_pairs& pr, const float* slot_out,
               float* grad_part, int32_t* status, int grid, cudaStream_t st) {
    if (net.xd != XD || net.h1 != H || net.h2 != H || net.d2mask != D2 || net.act != ACT) return 1;
    if (mode == 2) return FBP_OK;
    return launch_adjoint_tc<XD, H, D2, ACT>(net, x, pr, slot_out, grad_part, status, grid, st);
}

#define FBP_TC_ADJ_TRY(XD, H, D2, ACT)                                                              \
    {                                                                                               \
        int r_ = tc_adj_try<XD, H, D2, ACT>(mode, *net, x, *pr, slot_out, grad_part, status, grid, st);  \
        if (r_ != 1) return r_;                                                                     \
    }

}  // namespace fbp
