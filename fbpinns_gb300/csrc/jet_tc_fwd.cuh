// Tensor-core (tcgen05, 3xTF32) per-pair forward jets for networks with two
// hidden layers of H = 16 or 32 neurons.
//
// Layer 2 of the jet, z_c[k] = sum_n W2[k][n] v_c[n] (+ b2[k] for c = 0), is J
// GEMMs per tile of 128 pairs.  The layer-1 jet components factor as v_0 = a,
// v_{1+d} = tp cw[:, d] and v_{1+xd+s} = tpp c2_s (a, tp, tpp = the activation
// and its first two derivatives at the neuron's pre-activation; cw = W1 / sd,
// c2_s the sum of cw[:, d]^2 over the dims of second-derivative slot s), so
// the pair-dependent operands are only a, tp and tpp / k2 (TcAct), and the
// per-neuron scales are in B_c = W2 diag(f_c).  In shared memory the operands of a
// tile take 48 or 96 KB and an MMA at least 40 cycles to read them; here they
// live in tensor memory, written by the threads of the pair (H / 8 per pair,
// eight neurons each; two CTAs of 256 threads or one of 512 per SM), where an
// MMA takes N/2 cycles.  Each thread finishes its neurons' tanh jets and leaves
// its part of the output layer's sums in shared memory; one of the pair's
// threads (the groups take turns by tile) adds the parts, applies
// unnormalisation and window and writes the record.  The z accumulators are
// double-buffered where tensor memory suffices (H = 32: J <= 5): tile t's MMAs then run
// during the jets of tile t - 1.
//
// What bounds it: issue slots (50% busy with 16 warps) of the jets and splits,
// and the tile's two barriers.  Measured on a GB300: 2.34e6 pairs of 2-16-16-1
// networks, J = 4, 0.161 -> 0.137 ms (operands in shared memory, one thread per
// pair); a training step of 4096 networks 2-32-32-1 on 2.1e6 points 11.9 ->
// 9.5 ms, of 900 networks 3-32-32-1 (J = 6) on 58^3 points 4.40 -> 3.15 ms, of
// 341 SIRENs or AdaptiveFCNs 2-16-16-1 on 65537 points 582 -> 570 and 530 -> 509
// us (FMA kernel before).
#pragma once

#include <algorithm>
#include <atomic>

#include "tc_ops.cuh"

namespace fbp {

template <class C>
struct TcFwd {
    static_assert(C::TWO && C::H1 == C::H2 && (C::H1 == 16 || C::H1 == 32), "tensor-core forward shape");
    static constexpr bool SINL = TcAct<C>::template SIN<false>;  // the tpp operand is a
    static constexpr int H = C::H1, J = C::J, XD = C::XD, NS = C::NS;
    static constexpr int NPT = H / 8, T = 128 * NPT;
    static constexpr int NA = NS > 0 ? 3 : 2, OP = 2 * H;
    static constexpr int COLS = 16 * H;
    static constexpr int NBUF = NA * OP + 2 * J * H <= COLS ? 2 : 1;
    static_assert(NA * OP + NBUF * J * H <= COLS, "TMEM columns");
    static constexpr int cZ = NA * OP;
    // registers per thread: 112 (of the 128 that the CTAs' threads could have)
    // leave a CTA of the list kernels of the next batch room beside the resident
    // CTAs.  16381 points, levels 1..8: step 161 us, with 128 registers 178;
    // 2^18 points, levels 1..32: 2045 us at 112, 2048 at 128, 2066 at 104
    static constexpr int REGS = 112;
};

template <class C>
struct TcFwdSmem {
    using A = TcFwd<C>;
    float b[2][A::J * A::H * A::H];  // B_c (hi, lo): component c's rows k at c H + k, K = n
    float part[A::NPT][A::J][128];   // output-layer sums of each group's neurons
    float win[A::XD][3][128];        // 1D window factors
    uint64_t mbar;
    uint32_t tmem_base;
};

// GEMM 1's operand o, issued by one thread (small products first).
template <class C, int O>
__device__ __forceinline__ void tc_fwd_issue(uint32_t tmem, uint32_t zcol, uint32_t b_hi, uint32_t b_lo) {
    using A = TcFwd<C>;
    constexpr int H = A::H, c0 = O == 0 ? 0 : (O == 1 ? 1 : 1 + A::XD), nc = O == 0 ? 1 : (O == 1 ? A::XD : A::NS);
    constexpr uint32_t idesc = umma_idesc_tf32(128, nc * H), rows = (uint32_t)(c0 * (H / 8)) * KMajor<H>::SBO;
    const uint32_t d = tmem + zcol + c0 * H, a = tmem + (A::SINL && O == 2 ? 0 : O) * A::OP;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int ks = 0; ks < H / 8; ++ks)
            umma_tf32_ta(d, a + (p == 0 ? H : 0) + 8 * ks,
                         umma_desc((p == 1 ? b_lo : b_hi) + rows + ks * 256, KMajor<H>::LBO, KMajor<H>::SBO), idesc,
                         p + ks > 0);
}

template <class C>
__global__ void __maxnreg__(TcFwd<C>::REGS) forward_pairs_tm_kernel(fbp_net net, const float* __restrict__ x,
                                                                           fbp_pairs pr, float* __restrict__ pair_out,
                                                                           int32_t* __restrict__ status) {
    using A = TcFwd<C>;
    using F = TcAct<C>;
    constexpr int J = C::J, XD = C::XD, NS = C::NS, H = A::H, RS = rec_stride(J), NPT = A::NPT, NA = A::NA;
    __shared__ SParams<C> S;
    __shared__ int s_item;
    extern __shared__ float4 dyn_smem[];
    TcFwdSmem<C>& T = *reinterpret_cast<TcFwdSmem<C>*>(dyn_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = warp >> 2, r = (warp & 3) * 32 + lane, n0 = 8 * h;  // neurons [n0, n0 + 8) of the tile's pair r
    const uint32_t mbar = smem_u32(&T.mbar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(NA) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&T.tmem_base)),
                     "r"(A::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = T.tmem_base;
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)n0;  // this thread's lane and columns
    const uint32_t bh = smem_u32(&T.b[0][0]), bl = smem_u32(&T.b[1][0]);
    // test hook: no MMAs are issued, so the first wait runs out (short limit)
    const bool test_no_mma = (*(volatile int32_t*)status & FBP_STATUS_TC_TEST_NO_MMA) != 0;
    const uint64_t wait_ns = test_no_mma ? TC_TEST_WAIT_NS : TC_WAIT_NS;
    uint32_t phase = 0;
    bool failed = false;
    const int nit = (int)min((int64_t)*pr.n_items, pr.items_cap);
    int next;  // the item after this one, claimed at this one's start (see first_item)
    for (int it = first_item(pr, &s_item); it < nit && !failed; it = next) {
        const int j = pr.items[3 * (size_t)it], beg = pr.items[3 * (size_t)it + 1], cnt = pr.items[3 * (size_t)it + 2];
        const float* __restrict__ w2g = net.theta + (size_t)j * C::P + C::oW2;
        constexpr int PT = H * H / A::T;
        float w2[PT];
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            int k, n;
            KMajor<H>::at(tid + e * A::T, k, n);
            w2[e] = w2g[k * H + n];
        }
        // pair indices and raw coordinates of the next tile to stage (prefetched)
        int pos_n = 0, pt_n = 0;
        float xr[XD] = {};
        auto fetch = [&](int t) {
            if (t < cnt) {
                const int4 rec = pair_rec(pr, beg + t);
                pos_n = rec.x;
                pt_n = rec.y;
            }
        };
        auto fetch_x = [&](int t) {
            if (t < cnt)
#pragma unroll
                for (int d = 0; d < XD; ++d) xr[d] = x[(size_t)pt_n * XD + d];
        };
        fetch(r);
        __syncthreads();
        if (tid == 0 && pr.item_ctr) s_item = atomicAdd(pr.item_ctr, 1);
        fetch_x(r);
        load_params<C, false>(S, net, j);
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            const int o = tid + e * A::T;
            int k, n;
            KMajor<H>::at(o, k, n);
#pragma unroll
            for (int c = 0; c < J; ++c) {
                const float f = c == 0 ? 1.0f : (c <= XD ? S.cw[n * XD + (c - 1)] : S.c2[n * NS + (c - 1 - XD)]);
                const float v = c > XD ? w2[e] * f * F::template k2<false>(act_o<C, false>(S, n)) : w2[e] * f;
                split_tf32_rn(v, T.b[0][c * H * H + o], T.b[1][c * H * H + o]);
            }
        }
        fence_async_smem();
        const int ntile = (cnt + 127) / 128;
        float xp[XD] = {};  // the tile before: normalised point, record index, activity
        int pos_p = 0;
        bool act_p = false;
        // tanh jets of this thread's neurons of a tile -> its part of the output layer
        auto jets = [&](int ti) {
            float acc[J][8];
#pragma unroll
            for (int c = 0; c < J; ++c) tmem_ld8(mine + A::cZ + (ti % A::NBUF) * J * H + c * H, acc[c]);
            tmem_wait_ld();
            float2 o2[J];
#pragma unroll
            for (int c = 0; c < J; ++c) o2[c] = dup2(0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = n0 + 2 * q;
                float2 z[J], g[J];
#pragma unroll
                for (int c = 0; c < J; ++c) z[c] = make_float2(acc[c][2 * q], acc[c][2 * q + 1]);
                z[0] = add2(z[0], *reinterpret_cast<const float2*>(&S.b2[k]));
                if (pr.zs && act_p) {  // the layer-2 z-jets for the adjoint (fbp_pairs.zs: rows c * H + k)
                    float* zs = pr.zs + beg + ti * 128 + r;
#pragma unroll
                    for (int c = 0; c < J; ++c) {
                        __stcs(zs + (size_t)(c * H + k) * pr.zs_cap, z[c].x);
                        __stcs(zs + (size_t)(c * H + k + 1) * pr.zs_cap, z[c].y);
                    }
                }
                float2 tp;
                F::template first<true>(S, k, z[0], g[0], tp);
#pragma unroll
                for (int d = 0; d < XD; ++d) g[1 + d] = mul2(tp, z[1 + d]);
                if constexpr (NS > 0) {
                    const float2 tpp = F::template second<true>(S, k, F::template m2<true>(g[0], tp));
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        float2 q2 = dup2(0.f);  // sum of z_d^2 over the slot's dims
                        bool first = true;
#pragma unroll
                        for (int d = 0; d < XD; ++d)
                            if ((C::slot_dims(s) >> d) & 1) {
                                q2 = first ? mul2(z[1 + d], z[1 + d]) : fma2(z[1 + d], z[1 + d], q2);
                                first = false;
                            }
                        g[1 + XD + s] = fma2(tp, z[1 + XD + s], mul2(tpp, q2));
                    }
                }
                const float2 w3 = *reinterpret_cast<const float2*>(&S.W3[k]);
#pragma unroll
                for (int c = 0; c < J; ++c) o2[c] = fma2(w3, g[c], o2[c]);
            }
#pragma unroll
            for (int c = 0; c < J; ++c) T.part[h][c][r] = o2[c].x + o2[c].y;
            if (h < XD) {
                float v = xp[0];
#pragma unroll
                for (int d = 1; d < XD; ++d) v = h == d ? xp[d] : v;
                float c0, c1, c2;
                window_1d<C>(S, h, v, c0, c1, c2);
                T.win[h][0][r] = c0;
                T.win[h][1][r] = c1;
                T.win[h][2][r] = c2;
            }
        };
        // the pair's record from the parts
        auto record = [&](int ti) {
            if (h != ti % NPT || !act_p) return;
            float c0[XD], c1[XD], c2[XD], u[J], w[J], rec[RS];
#pragma unroll
            for (int d = 0; d < XD; ++d) {
                c0[d] = T.win[d][0][r];
                c1[d] = T.win[d][1][r];
                c2[d] = T.win[d][2][r];
            }
            window_product<C>(S, c0, c1, c2, w);
#pragma unroll
            for (int c = 0; c < J; ++c) {
                float o = c == 0 ? S.b3 : 0.f;
#pragma unroll
                for (int g = 0; g < NPT; ++g) o += T.part[g][c][r];
                u[c] = o * S.sd_u;
            }
            u[0] += S.mu_u;
            product_jet<C>(u, w, rec);
#pragma unroll
            for (int c = 0; c < J; ++c) rec[J + c] = w[c];
#pragma unroll
            for (int c = 2 * J; c < RS; ++c) rec[c] = 0.f;
            float4* dst = reinterpret_cast<float4*>(pair_out + (size_t)pos_p * RS);
#pragma unroll
            for (int q = 0; q < RS / 4; ++q)
                dst[q] = make_float4(rec[4 * q], rec[4 * q + 1], rec[4 * q + 2], rec[4 * q + 3]);
        };
        // Per tile: stage, barrier, issue, then the previous tile's jets (two z
        // buffers) or record (one), wait for the MMAs, then the previous tile's
        // record or this tile's jets.  A operands are rewritten only after that
        // wait, a z buffer only by MMAs issued after the barrier that follows its
        // reads, and the parts of one tile only after their record.
        for (int ti = 0; ti < ntile; ++ti) {
            float xn[XD];
            const int pos = pos_n;
            const bool act = ti * 128 + r < cnt;
#pragma unroll
            for (int d = 0; d < XD; ++d) xn[d] = act ? (xr[d] - S.mu[d]) * S.inv_sd[d] : 0.f;
            fetch((ti + 1) * 128 + r);
            {
                float a[8], tp[8], tpp[8];
#pragma unroll
                for (int q = 0; q < 8; q += 2) {
                    const int n = n0 + q;
                    float2 z = *reinterpret_cast<const float2*>(&S.b1[n]);
#pragma unroll
                    for (int d = 0; d < XD; ++d)
                        z = fma2(make_float2(S.W1[n * XD + d], S.W1[(n + 1) * XD + d]), dup2(xn[d]), z);
                    float2 av, t1;
                    F::template first<false>(S, n, z, av, t1);
                    a[q] = av.x, a[q + 1] = av.y;
                    tp[q] = t1.x, tp[q + 1] = t1.y;
                    if constexpr (NS > 0 && !A::SINL) {
                        const float2 t2 = F::template m2<false>(av, t1);
                        tpp[q] = t2.x, tpp[q + 1] = t2.y;
                    }
                }
                tmem_st_split8(mine, H, a);
                tmem_st_split8(mine + A::OP, H, tp);
                if constexpr (NS > 0 && !A::SINL) tmem_st_split8(mine + 2 * A::OP, H, tpp);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
            if (lane == 0 && warp < NA && !test_no_mma) {
                const uint32_t zc = A::cZ + (ti % A::NBUF) * J * H;
                if (warp == 0) tc_fwd_issue<C, 0>(tmem, zc, bh, bl);
                if (warp == 1) tc_fwd_issue<C, 1>(tmem, zc, bh, bl);
                if constexpr (NA > 2)
                    if (warp == 2) tc_fwd_issue<C, NA - 1>(tmem, zc, bh, bl);
                umma_commit(mbar);
            }
            __syncwarp();
            fetch_x((ti + 1) * 128 + r);
            if (ti > 0) {
                if constexpr (A::NBUF == 2) jets(ti - 1);
                else record(ti - 1);
            }
            failed = __syncthreads_or(warp == A::NA && !mbar_wait_warp(mbar, phase, wait_ns, lane));  // the verdict is CTA-uniform
            if (failed) break;
            phase ^= 1u;
            tc_fence_after();
            if constexpr (A::NBUF == 2) {
                if (ti > 0) record(ti - 1);
            }
#pragma unroll
            for (int d = 0; d < XD; ++d) xp[d] = xn[d];
            pos_p = pos;
            act_p = act;
            if constexpr (A::NBUF == 1) jets(ti);
        }
        if (failed) break;
        if constexpr (A::NBUF == 2) {
            __syncthreads();  // the parts of the tile before the last have been read
            jets(ntile - 1);
        }
        next = pr.item_ctr ? s_item : it + (int)gridDim.x;
        __syncthreads();
        record(ntile - 1);
    }
    if (failed) {
        if (tid == 0) atomicOr(status, FBP_STATUS_TC_TIMEOUT);
        mbar_wait_bounded(mbar, phase, wait_ns);  // let the timed-out MMAs finish
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A::COLS) : "memory");
}

template <int XD, int H, int D2, int ACT>
int launch_forward_tm(const fbp_net& net, const float* x, const fbp_pairs& pr, float* pair_out, int32_t* status,
                      int grid, cudaStream_t st) {
    using C = TcCfg<Cfg<XD, H, H, D2, ACT>>;
    FBP_REQUIRE(net.nparam == C::P, FBP_ERR_INVALID, "forward_tc: nparam %d != %d for this shape", net.nparam, C::P);
    // 512 / COLS CTAs per SM share its tensor memory (a further one would wait
    // in tcgen05.alloc); enough shared memory is asked for that no more fit
    constexpr int res = 512 / TcFwd<C>::COLS;
    const size_t shm = std::max(sizeof(TcFwdSmem<C>), (size_t)(228 / (res + 1) + 2) * 1024);
    static std::atomic<bool> attr_set[FBP_MAX_DEVICES] = {};  // set once per device (setting it twice is harmless)
    const int dev = current_device();
    if (!attr_set[dev].load()) {
        FBP_CUDA_CHECK(cudaFuncSetAttribute(forward_pairs_tm_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)shm));
        attr_set[dev].store(true);
    }
    if (grid <= 0) grid = (int)std::min<int64_t>(res * sm_count(), std::max<int64_t>(pr.items_cap, 1));
    if (pr.item_ctr) FBP_CUDA_CHECK(cudaMemsetAsync(pr.item_ctr, 0, sizeof(int32_t), st));
    forward_pairs_tm_kernel<C><<<grid, TcFwd<C>::T, shm, st>>>(net, x, pr, pair_out, status);
    FBP_LAUNCH_CHECK();
    return FBP_OK;
}

template <int XD, int H, int D2, int ACT>
int tm_try(int mode, const fbp_net& net, const float* x, const fbp_pairs& pr, float* pair_out, int32_t* status,
           int grid, cudaStream_t st) {
    if (net.xd != XD || net.h1 != H || net.h2 != H || net.d2mask != D2 || net.act != ACT) return 1;
    if (mode == 2) return FBP_OK;
    return launch_forward_tm<XD, H, D2, ACT>(net, x, pr, pair_out, status, grid, st);
}

}  // namespace fbp

#define FBP_TM_TRY(XD, H, D2, ACT)                                                             \
    {                                                                                          \
        int r_ = fbp::tm_try<XD, H, D2, ACT>(mode, *net, x, *pr, pair_out, status, grid, st);   \
        if (r_ != 1) return r_;                                                                \
    }
