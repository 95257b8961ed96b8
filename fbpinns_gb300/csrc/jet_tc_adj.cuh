// Tensor-core (tcgen05, 3xTF32) per-pair adjoint for networks with two hidden
// layers of equal width H = 16 or 32 and tanh, sin or adaptive activations
// (TcAct; written for tanh below).
//
// Of the adjoint's three layer-2 contractions, two have the pairs as rows and
// run on the tensor cores with the pair-dependent operand in tensor memory
// (the thread of a pair writes its own TMEM lane, so it costs no shared-memory
// traffic, and an MMA with A in TMEM takes N/2 cycles where one with A in
// shared memory takes at least 40):
//   GEMM 1  z_c = B_c v      B_c = W2 diag(f_c), v = a, tp or tpp of layer 1,
//           f_c = 1, W1[:, d] / sd_d, or the slot's sum of their squares
//   GEMM 2  T_0 = W2^T z2bar_0, T_1 = sum_d B_{1+d}^T z2bar_{1+d},
//           T_2 = sum_s B_s^T z2bar_s
// With T the layer-1 adjoint is z1bar = T_0 tp + T_1 tpp + T_2 tppp per neuron
// (tpp = -2 a tp with the -2 in the B operands); vbar is not formed.  The third contraction sums over the pairs,
//   S_c[k][n] = sum_pairs z2bar_c[k] m_c[n],   m = a, tp or tpp,
// and runs on warp-level MMAs (mma.sync, 3xTF32) from shared-memory rows while
// GEMM 2 is under way: tcgen05 would want at least 64 rows (c, k) by all three
// m, so that two thirds of its products are thrown away, with both operands
// split and transposed in shared memory (21 cycles per pair at H = 32, J = 4,
// against 24); packed FP32 FMAs need 1.1 words of shared memory per FMA pair
// and lane, over twice what it delivers (0.465 ms instead of 0.373 at
// 2.34e6 pairs, H = 16).  From S follow, once per work item,
//   W2bar = sum_c f_c S_c   and the tangent part of W1bar,
//   sum_pairs cwbar_d[n] = sum_k W2[k][n] (S_{1+d} + 2 cw_d sum_{s with d} S_s).
//
// A tile is 128 pairs; NPT = H / 8 threads share a pair (eight neurons each),
// so a CTA has 256 or 512 threads, two CTAs or one fill an SM's tensor memory,
// and 16 warps are resident.  The sums over pairs stay in registers for the
// whole work item (S_c as 4 x 2 blocks per lane, the biases', W3's and W1's
// value part per thread) and are reduced once, in a fixed order.
//
// What bounds it: issue slots (51% busy at H = 16, 43% at H = 32: elementwise
// jets, splits, the S_c loop) with 16 warps to hide the tiles' barriers; for
// H = 32 also the warp-level MMAs of S_c (24 cycles per pair at J = 4).
// Measured on a GB300, against the FMA adjoint (jet.cuh): 2.34e6 pairs of
// 2-16-16-1 networks, J = 4, 0.466 -> 0.337 ms; a training step of 4096
// networks 2-32-32-1 on 2.1e6 points 17.0 -> 11.9 ms, of 900 networks 3-32-32-1
// (J = 6) on 58^3 points 6.44 -> 4.40 ms with the same forward; of 341 SIRENs
// 2-16-16-1 on 65537 points 815 -> 582 us, of as many AdaptiveFCNs 840 -> 530 us
// (the parameters of adaptive activations need no sums over pairs of their own:
// their gradients follow from the weights', at the item's end).
//
// Waits on the MMA-completion mbarriers are bounded: on a time-out the kernel
// records FBP_STATUS_TC_TIMEOUT, stops, waits once more and frees its TMEM.
#pragma once

#include "tc_ops.cuh"

namespace fbp {

template <class C>
struct TcAdj {
    static_assert(C::TWO && C::H1 == C::H2 && (C::H1 == 16 || C::H1 == 32) && C::J <= 6, "tensor-core adjoint shape");
    static constexpr int H = C::H1, J = C::J, XD = C::XD, NS = C::NS, E = C::EXTRA;
    static constexpr bool SINL = TcAct<C>::template SIN<false>;
    static constexpr int NPT = H / 8;      // threads per pair
    static constexpr int T = 128 * NPT;    // threads per CTA
    static constexpr int NW = T / 32;
    // the first second-derivative slot sums more than one dim
    static constexpr bool SUMS = NS > 0 && (C::slot_dims(0) & (C::slot_dims(0) - 1)) != 0;
    static constexpr int NA = NS > 0 ? 3 : 2;  // A operands a, tp (, tpp); also the GEMM 2 groups
    static constexpr int OP = 2 * H;           // TMEM columns of an operand: hi, lo
    // TMEM columns: [A operands | z | (z2bar operands past the NA-th) | T].  z2bar
    // operands 0 .. NA-1 take the A operands' columns (free once GEMM 1 is
    // done); the others follow z where the columns suffice, else they take z's
    // own columns after a barrier (OVER).
    static constexpr int COLS = 16 * H;
    static constexpr int MORE = (J > NA ? J - NA : 0) * OP;
    static constexpr bool OVER = NA * OP + J * H + MORE + NA * H > COLS;
    static constexpr int cZ = NA * OP;
    static constexpr int cM = OVER ? cZ : cZ + J * H;
    static constexpr int cT = OVER ? cZ + J * H : cM + MORE;
    static_assert(cT + NA * H <= COLS && (!OVER || MORE <= J * H), "TMEM columns");
    __host__ __device__ static constexpr int zcol(int c) { return c < NA ? c * OP : cM + (c - NA) * OP; }
    // shared-memory rows: z2bar [c][k] (row stride 4 mod 32 words: 16-byte
    // accesses of eight consecutive rows hit different banks), a [n]
    static constexpr int ZS = (J * H + 31) / 32 * 32 + 4, AS = H + 4;
    // S_c blocks: a warp has 16 k x 8 NQ n (NQ = 1 where J blocks of two would
    // not fit the registers); SUB warps cover H x H, PG groups of warps split
    // the tile's pairs
    static constexpr int NQ = J > 4 ? 1 : 2;
    static constexpr int KB = H / 16, SUB = KB * (H / (8 * NQ)), PG = NW / SUB, PPG = 128 / PG;
    // per-thread sums over the item's pairs of 8 neurons: W3, b2, b1, W1's value part
    static constexpr int iW3 = 0, iB2 = 1, iB1 = 2, iW1 = 3, NSUM = 3 + XD;
    // those from iB1 on are kept in shared memory between tiles where it has
    // the room (as float4, conflict-free), else in registers
    static constexpr int NST = 2 * (NSUM - iB1);
    static constexpr int BASE = 4 * (4 * J * H * H + 128 * (ZS + AS * (SINL ? 2 : 1)) + 2 * (XD + J) * 128 +
                                     4 * NPT * 8 * NSUM);
    static constexpr bool STASH = BASE + NST * T * 16 <= (H == 16 ? 111 : 222) * 1024;
};

template <class C>
struct TcAdjSmem {
    using A = TcAdj<C>;
    float b1[2][A::J * A::H * A::H];  // GEMM 1 B (hi, lo): component c's rows k at c H + k, K = n
    float b2[2][A::J * A::H * A::H];  // GEMM 2 B: component c's H x H matrix, rows n, K = k
    float zb[128 * A::ZS];            // z2bar rows; at the item's end the S_c of the pair groups
    float a1[128 * A::AS];            // layer-1 activations
    float tp1[A::SINL ? 128 * A::AS : 4];  // and their first derivatives where those do not follow from them
    float xo[2][A::XD + A::J][128];   // per pair of this and the next tile: normalised point, o-bar jet
    float red[4 * A::NPT][8 * A::NSUM];  // per warp: the item's sums over its lanes
    float4 stash[A::STASH ? A::NST : 1][A::STASH ? A::T : 1];
    float red3[4];
    float redx[2][A::H];  // sums of W2 W2-bar over k and over n (adaptive activations)
    uint64_t mbar[2];
    uint32_t tmem_base;
};

// The MMAs of one operand group, issued by one thread: GEMM 1's operand o
// (value, tangents or second derivatives) or GEMM 2's group g.  Small
// products first, so that the large ones are added (and rounded) last.
template <class C, int O>
__device__ __forceinline__ void tc_adj_issue1(uint32_t tmem, uint32_t b_hi, uint32_t b_lo) {
    using A = TcAdj<C>;
    constexpr int H = A::H, c0 = O == 0 ? 0 : (O == 1 ? 1 : 1 + A::XD), nc = O == 0 ? 1 : (O == 1 ? A::XD : A::NS);
    constexpr uint32_t idesc = umma_idesc_tf32(128, nc * H), rows = (uint32_t)(c0 * (H / 8)) * KMajor<H>::SBO;
    const uint32_t d = tmem + A::cZ + c0 * H, a = tmem + (A::SINL && O == 2 ? 0 : O) * A::OP;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int ks = 0; ks < H / 8; ++ks)
            umma_tf32_ta(d, a + (p == 0 ? H : 0) + 8 * ks,
                         umma_desc((p == 1 ? b_lo : b_hi) + rows + ks * 256, KMajor<H>::LBO, KMajor<H>::SBO), idesc,
                         p + ks > 0);
}

template <class C, int G>
__device__ __forceinline__ void tc_adj_issue2(uint32_t tmem, uint32_t b_hi, uint32_t b_lo) {
    using A = TcAdj<C>;
    constexpr int H = A::H, c0 = G == 0 ? 0 : (G == 1 ? 1 : 1 + A::XD), nc = G == 0 ? 1 : (G == 1 ? A::XD : A::NS);
    constexpr uint32_t idesc = umma_idesc_tf32(128, H);
    const uint32_t d = tmem + A::cT + G * H;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int c = c0; c < c0 + nc; ++c)
#pragma unroll
            for (int ks = 0; ks < H / 8; ++ks)
                umma_tf32_ta(d, tmem + A::zcol(c) + (p == 0 ? H : 0) + 8 * ks,
                             umma_desc((p == 1 ? b_lo : b_hi) + c * H * H * 4 + ks * 256, KMajor<H>::LBO,
                                       KMajor<H>::SBO),
                             idesc, p + (c - c0) + ks > 0);
}

// Runs F<0>, F<1> (, F<2>) on lane 0 of warps 0, 1 (, 2): one thread needs about
// 45 cycles per MMA it issues, so the groups go out in parallel.
#define FBP_TC_ISSUE(F, hi, lo, bar)                            \
    if (lane == 0 && warp < A::NA && !test_no_mma) {            \
        if (warp == 0) F<C, 0>(tmem, hi, lo);                   \
        if (warp == 1) F<C, 1>(tmem, hi, lo);                   \
        if constexpr (A::NA > 2)                                \
            if (warp == 2) F<C, A::NA - 1>(tmem, hi, lo);       \
        umma_commit(bar);                                       \
    }

template <class C>
__global__ void __launch_bounds__(TcAdj<C>::T, 32 / C::H1) adjoint_pairs_tc_kernel(fbp_net net,
                                                                                    const float* __restrict__ x,
                                                                                    fbp_pairs pr,
                                                                                    const float* __restrict__ slot_out,
                                                                                    float* __restrict__ grad_part,
                                                                                    int32_t* __restrict__ status) {
    using A = TcAdj<C>;
    using F = TcAct<C>;
    constexpr int J = C::J, XD = C::XD, NS = C::NS, E = A::E, H = A::H, RS = rec_stride(J), NPT = A::NPT, NA = A::NA;
    static_assert(A::PG * J * H * H <= 128 * A::ZS && (XD + 2) * H * (H + 1) <= 128 * A::ZS, "S_c fit the z2bar rows");
    __shared__ SParams<C> S;
    __shared__ int s_item;
    extern __shared__ float4 dyn_smem[];
    TcAdjSmem<C>& T = *reinterpret_cast<TcAdjSmem<C>*>(dyn_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = warp >> 2, r = (warp & 3) * 32 + lane;  // neurons [8h, 8h + 8) of the tile's pair r
    const int n0 = 8 * h;
    const uint32_t mbar1 = smem_u32(&T.mbar[0]), mbar2 = smem_u32(&T.mbar[1]);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar1), "r"(NA) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar2), "r"(NA) : "memory");
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
    pdl_wait();
    const uint32_t tmem = T.tmem_base;
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)n0;  // this thread's lane and columns
    const uint32_t b1h = smem_u32(&T.b1[0][0]), b1l = smem_u32(&T.b1[1][0]);
    const uint32_t b2h = smem_u32(&T.b2[0][0]), b2l = smem_u32(&T.b2[1][0]);
    const bool test_no_mma = (*(volatile int32_t*)status & FBP_STATUS_TC_TEST_NO_MMA) != 0;
    const uint64_t wait_ns = test_no_mma ? TC_TEST_WAIT_NS : TC_WAIT_NS;
    // this lane's block of the S_c loop
    const int sk = 16 * (warp % A::SUB % A::KB) + (lane >> 2), sn = 8 * A::NQ * (warp % A::SUB / A::KB);
    const int sp = (warp / A::SUB) * A::PPG;  // first pair of the warp's group
    uint32_t phase = 0;
    bool failed = false;
    const int nit = (int)min((int64_t)*pr.n_items, pr.items_cap);
    int next;  // the item after this one, claimed at this one's start (see first_item)
    for (int it = first_item(pr, &s_item); it < nit && !failed; it = next) {
        const int j = pr.items[3 * (size_t)it], beg = pr.items[3 * (size_t)it + 1], cnt = pr.items[3 * (size_t)it + 2];
        const float* __restrict__ w2g = net.theta + (size_t)j * C::P + C::oW2;
        constexpr int PT = H * H / A::T;  // entries of W2 per thread
        int4 rec = make_int4(0, 0, -1, 0);
        float xr[XD] = {}, w2[PT];
        float4 sd[(J + 3) / 4] = {};
        if (h == 0 && r < cnt) rec = pair_rec(pr, beg + r);
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            int k, n;
            KMajor<H>::at(tid + e * A::T, k, n);
            w2[e] = w2g[k * H + n];
        }
        __syncthreads();
        if (tid == 0 && pr.item_ctr) s_item = atomicAdd(pr.item_ctr, 1);
        // pair t of the item: normalised point and o-bar jet (from the seeds of its slot)
        auto prep = [&](int buf, bool act) {
            float xn[XD], ob[J];
#pragma unroll
            for (int d = 0; d < XD; ++d) xn[d] = act ? (xr[d] - S.mu[d]) * S.inv_sd[d] : 0.f;
#pragma unroll
            for (int c = 0; c < J; ++c) ob[c] = 0.f;
            if (act) {
                float w[J], nb[J], ub[J];
                window_jet<C>(S, xn, w);
                const bool ok = rec.z >= 0 && rec.z < pr.slots_cap;  // overflowed slots carry no seed
#pragma unroll
                for (int c = 0; c < J; ++c) {
                    const float4 v = sd[c / 4];
                    nb[c] = !ok ? 0.f : (c % 4 == 0 ? v.x : c % 4 == 1 ? v.y : c % 4 == 2 ? v.z : v.w);
                }
                product_jet_adj<C>(nb, w, ub);
#pragma unroll
                for (int c = 0; c < J; ++c) ob[c] = ub[c] * S.sd_u;
            }
#pragma unroll
            for (int d = 0; d < XD; ++d) T.xo[buf][d][r] = xn[d];
#pragma unroll
            for (int c = 0; c < J; ++c) T.xo[buf][XD + c][r] = ob[c];
        };
        auto fetch = [&]() {
#pragma unroll
            for (int d = 0; d < XD; ++d) xr[d] = x[(size_t)rec.y * XD + d];
            const bool ok = rec.z >= 0 && rec.z < pr.slots_cap;
            const float4* src = reinterpret_cast<const float4*>(slot_out + (size_t)(ok ? rec.z : 0) * RS);
#pragma unroll
            for (int q = 0; q < (J + 3) / 4; ++q) sd[q] = src[q];
        };
        if (h == 0 && r < cnt) fetch();
        load_params<C, false>(S, net, j);
        if (h == 0) prep(0, r < cnt);  // the first tile's pairs
        // B operands
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            const int o = tid + e * A::T;
            int k, n;
            KMajor<H>::at(o, k, n);
            const int ot = KMajor<H>::off(n, k);
#pragma unroll
            for (int c = 0; c < J; ++c) {
                const float f = c == 0 ? 1.0f : (c <= XD ? S.cw[n * XD + (c - 1)] : S.c2[n * NS + (c - 1 - XD)]);
                // k2 = tpp / m2 goes with the second-derivative operands of GEMM 1
                // and the tangents of GEMM 2 (T_1 tpp), o^2 with its second
                // derivatives (T_2 tppp)
                const float o1 = act_o<C, false>(S, n), k2 = F::template k2<false>(o1), v = w2[e] * f;
                const float v1 = c > XD ? v * k2 : v, v2 = c == 0 ? v : (c <= XD ? v * k2 : v * (o1 * o1));
                split_tf32_rn(v1, T.b1[0][c * H * H + o], T.b1[1][c * H * H + o]);    // rows k, K = n
                split_tf32_rn(v2, T.b2[0][c * H * H + ot], T.b2[1][c * H * H + ot]);  // rows n, K = k
            }
        }
        if (h == 1 && 128 + r < cnt) rec = pair_rec(pr, beg + 128 + r);  // the second tile's pairs
        fence_async_smem();
        float sacc[J][A::NQ][4];  // S_c, 16 k x 8 NQ n as MMA accumulators (c > XD: over m2 = tpp / k2)
        float2 sum[A::NSUM][4];  // see TcAdj
        float g3b = 0.f;
#pragma unroll
        for (int c = 0; c < J; ++c)
#pragma unroll
            for (int q = 0; q < A::NQ; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) sacc[c][q][i] = 0.f;
#pragma unroll
        for (int i = 0; i < A::NSUM; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[i][q] = dup2(0.f);
        auto stash = [&](bool load) {  // the sums from iB1 on, from / to shared memory
#pragma unroll
            for (int i = A::iB1; i < A::NSUM; ++i) {
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    float4& w = T.stash[A::STASH ? 2 * (i - A::iB1) + b : 0][A::STASH ? tid : 0];
                    if (load) {
                        const float4 v = w;
                        sum[i][2 * b] = make_float2(v.x, v.y);
                        sum[i][2 * b + 1] = make_float2(v.z, v.w);
                    } else {
                        w = make_float4(sum[i][2 * b].x, sum[i][2 * b].y, sum[i][2 * b + 1].x, sum[i][2 * b + 1].y);
                    }
                }
            }
        };
        if constexpr (A::STASH) stash(false);
        __syncthreads();
        const int ntile = (cnt + 127) / 128;
        for (int ti = 0; ti < ntile; ++ti) {
            const int buf = ti & 1;
            float* zrow = &T.zb[r * A::ZS + n0];
            float* arow = &T.a1[r * A::AS + n0];
            // the next tile's pairs: the groups of threads take turns; the record was
            // fetched a tile ago
            const bool mypre = ti + 1 < ntile && h == (ti + 1) % NPT, nact = (ti + 1) * 128 + r < cnt;
            if (mypre && nact) fetch();
            // ---- layer 1 of this thread's neurons -> A operands and the a row ----
            {
                float a[8], tp[8], tpp[8];
                float xn[XD];
#pragma unroll
                for (int d = 0; d < XD; ++d) xn[d] = T.xo[buf][d][r];
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
                *reinterpret_cast<float4*>(arow) = make_float4(a[0], a[1], a[2], a[3]);
                *reinterpret_cast<float4*>(arow + 4) = make_float4(a[4], a[5], a[6], a[7]);
                if constexpr (A::SINL) {
                    float* trow = &T.tp1[r * A::AS + n0];
                    *reinterpret_cast<float4*>(trow) = make_float4(tp[0], tp[1], tp[2], tp[3]);
                    *reinterpret_cast<float4*>(trow + 4) = make_float4(tp[4], tp[5], tp[6], tp[7]);
                }
                tmem_st_split8(mine, H, a);
                tmem_st_split8(mine + A::OP, H, tp);
                if constexpr (NS > 0 && !A::SINL) tmem_st_split8(mine + 2 * A::OP, H, tpp);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
            FBP_TC_ISSUE(tc_adj_issue1, b1h, b1l, mbar1)
            __syncwarp();
            if (mypre) prep(buf ^ 1, nact);
            // (a time-out counts at the tile's last barrier, where the verdict is CTA-uniform)
            bool late = !mbar_wait_warp(mbar1, phase, wait_ns, lane);
            tc_fence_after();
            // ---- tanh jets of layer 2 and their adjoint -> z2bar ----
            {
                float ob[J];
#pragma unroll
                for (int c = 0; c < J; ++c) ob[c] = T.xo[buf][XD + c][r];
                if (h == 0) g3b += ob[0];
                // eight neurons at a time, or four, with z2bar split for TMEM from its row
                // afterwards, where z's columns are taken by z2bar (that wait for every
                // thread's z would keep all J x 8 in registers) and where a slot sums
                // several dims (its z_d^2 and P take registers too).  Steps in us, eight
                // and four: Laplacian jets, Helmholtz 8452 8399, SIREN 528 522, Poisson
                // of 16381 points 119 117.5; u_xx alone, Burgers 69.0 69.8
                constexpr int NH = A::OVER || A::SUMS ? 4 : 8;
#pragma unroll
                for (int half = 0; half < 8 / NH; ++half) {
                    float acc[J][NH];
#pragma unroll
                    for (int c = 0; c < J; ++c) {
                        if constexpr (NH == 8) tmem_ld8(mine + A::cZ + c * H, acc[c]);
                        else tmem_ld4(mine + A::cZ + c * H + half * NH, acc[c]);
                    }
                    tmem_wait_ld();
#pragma unroll
                    for (int qq = 0; qq < NH / 2; ++qq) {
                        const int q = half * (NH / 2) + qq, k = n0 + 2 * q;
                        float2 z[J];
#pragma unroll
                        for (int c = 0; c < J; ++c) z[c] = make_float2(acc[c][2 * qq], acc[c][2 * qq + 1]);
                        z[0] = add2(z[0], *reinterpret_cast<const float2*>(&S.b2[k]));
                        float2 a, tp;
                        F::template first<true>(S, k, z[0], a, tp);
                        const float2 tpp = F::template second<true>(S, k, F::template m2<true>(a, tp));
                        const float2 tppp = F::template third<true>(S, k, tp);
                        // the sensitivities of sigma' and sigma'' over W3: P = sum_d ob_d z_d +
                        // sum_s ob_s z_s, Q = sum_s ob_s sum_d z_d^2; then W3-bar += ob_0 a +
                        // tp P + tpp Q, z2bar_0 = W3 (ob_0 tp + tpp P + tppp Q), z2bar_d =
                        // W3 (ob_d tp + 2 ob_s tpp z_d), z2bar_s = W3 ob_s tp
                        const float2 w3 = *reinterpret_cast<const float2*>(&S.W3[k]);
                        const float2 wtp = mul2(w3, tp), w4 = mul2(dup2(2.0f), mul2(w3, tpp));
                        float2 P = mul2(dup2(ob[1]), z[1]), Q = dup2(0.f), zb[J];
#pragma unroll
                        for (int d = 1; d < XD; ++d) P = fma2(dup2(ob[1 + d]), z[1 + d], P);
#pragma unroll
                        for (int d = 0; d < XD; ++d) zb[1 + d] = mul2(dup2(ob[1 + d]), wtp);
#pragma unroll
                        for (int s = 0; s < NS; ++s) {
                            const float2 os = dup2(ob[1 + XD + s]), o4 = mul2(os, w4);
                            float2 q2 = dup2(0.f);  // sum of z_d^2 over the slot's dims
                            bool first = true;
#pragma unroll
                            for (int d = 0; d < XD; ++d)
                                if ((C::slot_dims(s) >> d) & 1) {
                                    q2 = first ? mul2(z[1 + d], z[1 + d]) : fma2(z[1 + d], z[1 + d], q2);
                                    first = false;
                                    zb[1 + d] = fma2(o4, z[1 + d], zb[1 + d]);
                                }
                            P = fma2(os, z[1 + XD + s], P);
                            Q = s == 0 ? mul2(os, q2) : fma2(os, q2, Q);
                            zb[1 + XD + s] = mul2(os, wtp);
                        }
                        float2 s3 = fma2(tp, P, fma2(dup2(ob[0]), a, sum[A::iW3][q]));
                        float2 z0 = fma2(tpp, P, mul2(dup2(ob[0]), tp));
                        if constexpr (NS > 0) {
                            s3 = fma2(tpp, Q, s3);
                            z0 = fma2(tppp, Q, z0);
                        }
                        zb[0] = mul2(w3, z0);
                        sum[A::iW3][q] = s3;
                        sum[A::iB2][q] = add2(sum[A::iB2][q], zb[0]);
#pragma unroll
                        for (int c = 0; c < J; ++c) acc[c][2 * qq] = zb[c].x, acc[c][2 * qq + 1] = zb[c].y;
                    }
#pragma unroll
                    for (int c = 0; c < J; ++c) {
#pragma unroll
                        for (int i = 0; i < NH; i += 4)
                            *reinterpret_cast<float4*>(zrow + c * H + half * NH + i) =
                                make_float4(acc[c][i], acc[c][i + 1], acc[c][i + 2], acc[c][i + 3]);
                        if constexpr (NH == 8) tmem_st_split8(mine + A::zcol(c), H, acc[c]);
                    }
                }
                if constexpr (A::OVER) {
                    tc_fence_before();
                    __syncthreads();  // every thread has read its z
                    tc_fence_after();
                }
                if constexpr (NH == 4) {
#pragma unroll
                    for (int c = 0; c < J; ++c) {  // this thread's own row
                        const float4 u = *reinterpret_cast<const float4*>(zrow + c * H);
                        const float4 v = *reinterpret_cast<const float4*>(zrow + c * H + 4);
                        const float zc[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
                        tmem_st_split8(mine + A::zcol(c), H, zc);
                    }
                }
            }
            tmem_wait_st();
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
            FBP_TC_ISSUE(tc_adj_issue2, b2h, b2l, mbar2)
            __syncwarp();
            if (h == (ti + 2) % NPT && (ti + 2) * 128 + r < cnt) rec = pair_rec(pr, beg + (ti + 2) * 128 + r);
            // ---- S_c over the warp's pairs, eight at a time, while GEMM 2 runs ----
            // (K index t of the MMA is pair p + 2t, t + 4 pair p + 2t + 1: loads
            // without bank conflicts.  The MMA's sums are truncated, so each group
            // of eight pairs starts from zero and is added in FP32.)
            {
                auto split = [](float2 v, float* hi, float* lo) {
                    float2 a, b;
                    split2_tf32_rn(v, a, b);
                    hi[0] = a.x, hi[1] = a.y, lo[0] = b.x, lo[1] = b.y;
                };
                const int np = min(A::PPG, cnt - (ti * 128 + sp));
                const int p2 = sp + 2 * (lane & 3);
                const float* zr = &T.zb[p2 * A::ZS + sk];
                const float* ar = &T.a1[p2 * A::AS + sn + (lane >> 2)];
                const float* tr = A::SINL ? &T.tp1[p2 * A::AS + sn + (lane >> 2)] : ar;  // (read for sine only)
#pragma unroll 1
                for (int p = 0; p < np; p += 8, zr += 8 * A::ZS, ar += 8 * A::AS, tr += 8 * A::AS) {
                    float bh[NA][A::NQ][2], bl[NA][A::NQ][2];
#pragma unroll
                    for (int q = 0; q < A::NQ; ++q) {
                        const float2 a = make_float2(ar[8 * q], ar[A::AS + 8 * q]);
                        float2 tp;
                        if constexpr (A::SINL) {
                            tp = make_float2(tr[8 * q], tr[A::AS + 8 * q]);
                        } else {
                            float2 t = a;
                            if constexpr (E > 0) t = mul2(a, dup2(act_o<C, false>(S, sn + (lane >> 2) + 8 * q)));
                            tp = fma2(make_float2(-t.x, -t.y), t, dup2(1.0f));
                        }
                        split(a, bh[0][q], bl[0][q]);
                        split(tp, bh[1][q], bl[1][q]);
                        if constexpr (NS > 0 && !A::SINL) split(F::template m2<false>(a, tp), bh[NA - 1][q], bl[NA - 1][q]);
                    }
#pragma unroll
                    for (int c = 0; c < J; ++c) {
                        const int o = c == 0 ? 0 : (c <= XD ? 1 : (A::SINL ? 0 : NA - 1));
                        float ah[4], al[4];
                        split(make_float2(zr[c * H], zr[c * H + 8]), ah, al);
                        split(make_float2(zr[A::ZS + c * H], zr[A::ZS + c * H + 8]), ah + 2, al + 2);
#pragma unroll
                        for (int q = 0; q < A::NQ; ++q) {
                            float d[4];
                            mma_tf32<true>(d, al, bh[o][q]);
                            mma_tf32(d, ah, bl[o][q]);
                            mma_tf32(d, ah, bh[o][q]);
#pragma unroll
                            for (int i = 0; i < 4; i += 2) {
                                const float2 v = add2(make_float2(sacc[c][q][i], sacc[c][q][i + 1]), make_float2(d[i], d[i + 1]));
                                sacc[c][q][i] = v.x, sacc[c][q][i + 1] = v.y;
                            }
                        }
                    }
                }
            }
            late |= !mbar_wait_warp(mbar2, phase, wait_ns, lane);
            failed = __syncthreads_or(late);
            if (failed) break;
            phase ^= 1u;
            tc_fence_after();
            // ---- layer-1 adjoint: b1-bar and the value part of W1-bar ----
            {
                float tb[NA][8];
#pragma unroll
                for (int g = 0; g < NA; ++g) tmem_ld8(mine + A::cT + g * H, tb[g]);
                float xn[XD];
#pragma unroll
                for (int d = 0; d < XD; ++d) xn[d] = T.xo[buf][d][r];
                if constexpr (A::STASH) stash(true);
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int n = n0 + 2 * q;
                    const float2 a = *reinterpret_cast<const float2*>(arow + 2 * q);
                    const float2 t0 = make_float2(tb[0][2 * q], tb[0][2 * q + 1]);
                    const float2 t1 = make_float2(tb[1][2 * q], tb[1][2 * q + 1]);
                    const float2 t2 = NS > 0 ? make_float2(tb[NA - 1][2 * q], tb[NA - 1][2 * q + 1]) : dup2(0.f);
                    float2 tp, z1;
                    if constexpr (A::SINL) {
                        tp = *reinterpret_cast<const float2*>(&T.tp1[r * A::AS + n]);
                    } else {
                        float2 t = a;
                        if constexpr (E > 0) t = mul2(a, make_float2(act_o<C, false>(S, n), act_o<C, false>(S, n + 1)));
                        tp = fma2(make_float2(-t.x, -t.y), t, dup2(1.0f));
                    }
                    if constexpr (A::SINL) {
                        // z1bar = tp (T_0 - T_2) + a T_1, with the factors in B
                        z1 = fma2(a, t1, mul2(tp, add2(t0, make_float2(-t2.x, -t2.y))));
                    } else {
                        // z1bar = tp (T_0 + a T_1 + (4 - 6 tp) T_2)
                        z1 = fma2(a, t1, t0);
                        if constexpr (NS > 0) z1 = fma2(fma2(dup2(-6.0f), tp, dup2(4.0f)), t2, z1);
                        z1 = mul2(z1, tp);
                    }
                    sum[A::iB1][q] = add2(sum[A::iB1][q], z1);
#pragma unroll
                    for (int d = 0; d < XD; ++d) sum[A::iW1 + d][q] = fma2(z1, dup2(xn[d]), sum[A::iW1 + d][q]);
                }
                if constexpr (A::STASH) stash(false);
            }
        }
        if (failed) break;
        // ---- the item's gradient partial: sums over lanes, warps and pair groups in a fixed order ----
        float* dst = grad_part + (size_t)it * C::P;
        if constexpr (A::STASH) stash(true);
        {
#pragma unroll
            for (int i0 = 0; i0 < A::NSUM; i0 += 4) {
                constexpr int NS4 = A::NSUM;
                if (NS4 - i0 > 2) {
                    float v[32];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 w = i0 + i < NS4 ? sum[i0 + i < NS4 ? i0 + i : 0][q] : dup2(0.f);
                            v[8 * i + 2 * q] = w.x, v[8 * i + 2 * q + 1] = w.y;
                        }
                    warp_reduce_scatter<32>(v, lane);
                    if (8 * i0 + lane < 8 * NS4) T.red[warp][8 * i0 + lane] = v[0];
                } else {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 w = i0 + i < NS4 ? sum[i0 + i < NS4 ? i0 + i : 0][q] : dup2(0.f);
                            v[8 * i + 2 * q] = w.x, v[8 * i + 2 * q + 1] = w.y;
                        }
                    warp_reduce_scatter<16>(v, lane);
                    if (!(lane & 1) && 8 * i0 + (lane >> 1) < 8 * NS4) T.red[warp][8 * i0 + (lane >> 1)] = v[0];
                }
            }
            if (h == 0) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) g3b += __shfl_xor_sync(0xffffffffu, g3b, o);
                if (lane == 0) T.red3[warp] = g3b;
            }
        }
        // pair groups' S_c: [group][c][k][n]
#pragma unroll
        for (int c = 0; c < J; ++c)
#pragma unroll
            for (int q = 0; q < A::NQ; ++q) {
                float* p = &T.zb[((warp / A::SUB) * J + c) * H * H + sk * H + sn + 8 * q + 2 * (lane & 3)];
                *reinterpret_cast<float2*>(p) = make_float2(sacc[c][q][0], sacc[c][q][1]);
                *reinterpret_cast<float2*>(p + 8 * H) = make_float2(sacc[c][q][2], sacc[c][q][3]);
            }
        next = pr.item_ctr ? s_item : it + (int)gridDim.x;
        __syncthreads();
        float s[PT][J], w2bar[PT];
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            const int i = tid + e * A::T, n = i % H;
#pragma unroll
            for (int c = 0; c < J; ++c) {
                float v = 0.f;
#pragma unroll
                for (int g = 0; g < A::PG; ++g) v += T.zb[(g * J + c) * H * H + i];
                s[e][c] = c > XD ? F::template k2<false>(act_o<C, false>(S, n)) * v : v;
            }
            float v = s[e][0];
#pragma unroll
            for (int d = 0; d < XD; ++d) v = fmaf(S.cw[n * XD + d], s[e][1 + d], v);
#pragma unroll
            for (int q = 0; q < NS; ++q) v = fmaf(S.c2[n * NS + q], s[e][1 + XD + q], v);
            dst[C::oW2 + i] = v;
            w2bar[e] = v;
        }
        __syncthreads();
        // the tangent part of W1-bar: [d][k] rows of W2[k][n] (S_{1+d} + 2 cw_d sum_s S_s), summed over k
#pragma unroll
        for (int e = 0; e < PT; ++e) {
            const int i = tid + e * A::T, n = i % H, k = i / H;
            const float wkn = w2g[i];
#pragma unroll
            for (int d = 0; d < XD; ++d) {
                float v = 0.f;
#pragma unroll
                for (int q = 0; q < NS; ++q)
                    if ((C::slot_dims(q) >> d) & 1) v += s[e][1 + XD + q];
                v = fmaf(2.0f * S.cw[n * XD + d], v, s[e][1 + d]);
                T.zb[(d * H + n) * (H + 1) + k] = wkn * v;
            }
            if constexpr (E > 0) {  // W2 * W2-bar, for the sums over k and over n
                T.zb[(XD * H + n) * (H + 1) + k] = wkn * w2bar[e];
                T.zb[((XD + 1) * H + k) * (H + 1) + n] = wkn * w2bar[e];
            }
        }
        __syncthreads();
        for (int o = warp; o < H * (XD + (E > 0 ? 2 : 0)); o += A::NW) {  // one warp per (d, n)
            const int d = o / H, n = o - d * H;
            float v = lane < H ? T.zb[(d * H + n) * (H + 1) + lane] : 0.f;
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
            if (E > 0 && d >= XD) {
                if (lane == 0) T.redx[d - XD][n] = v;
            } else if (lane == 0) {
                const int w0 = (n >> 3) * 4, at = 8 * (A::iW1 + d) + (n & 7);
                float u = 0.f;
#pragma unroll
                for (int w = 0; w < 4; ++w) u += T.red[w0 + w][at];
                dst[C::oW1 + n * XD + d] = fmaf(v, S.inv_sd[d], u);
            }
        }
        for (int i = tid; i < 3 * H; i += A::T) {
            const int g = i / H, n = i - g * H, w0 = (n >> 3) * 4;
            float u = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) u += T.red[w0 + w][8 * g + (n & 7)];
            dst[(g == A::iW3 ? C::oW3 : (g == A::iB2 ? C::ob2 : C::ob1)) + n] = u;
        }
        if constexpr (E > 0) {
            // Activation parameters of sigma(z) = c f(o z): o scales the weights into
            // the neuron and c those out of it, so
            //   dL/do = (sum of W Wbar + b bbar of its layer) / o,
            //   dL/dc = (sum of W Wbar of the next layer) / c
            // AdaptiveFCN (c = a, o = 1/a): dL/da = dL/dc - o^2 dL/do.
            __syncthreads();  // the entries read back below are written
            if (tid < 2 * H) {
                const bool l2 = tid >= H;
                const int n = l2 ? tid - H : tid;
                float go, gc;
                if (l2) {
                    go = T.redx[1][n] + S.b2[n] * dst[C::ob2 + n];
                    gc = S.W3[n] * dst[C::oW3 + n];
                } else {
                    go = S.b1[n] * dst[C::ob1 + n];
#pragma unroll
                    for (int d = 0; d < XD; ++d) go = fmaf(S.W1[n * XD + d], dst[C::oW1 + n * XD + d], go);
                    gc = T.redx[0][n];
                }
                const float c = l2 ? act_c<C, true>(S, n) : act_c<C, false>(S, n);
                const float o = l2 ? act_o<C, true>(S, n) : act_o<C, false>(S, n);
                go /= o;
                gc /= c;
                float* gx = dst + (l2 ? C::oX2 : C::oX1) + n;
                if constexpr (C::ACT == FBP_ACT_ADAPTIVE_TANH) {
                    gx[0] = gc - o * o * go;
                } else {
                    gx[0] = gc;
                    gx[H] = go;
                }
            }
            if (tid < E) dst[C::oX3 + tid] = 0.f;  // the output layer's parameters are unused
        }
        if (tid == 0) dst[C::ob3] = (T.red3[0] + T.red3[1]) + (T.red3[2] + T.red3[3]);
    }
    if (failed) {
        if (tid == 0) atomicOr(status, FBP_STATUS_TC_TIMEOUT);
        // let the timed-out MMAs finish (phase is the same for both barriers or one behind)
        mbar_wait_bounded(mbar1, phase, wait_ns);
        mbar_wait_bounded(mbar2, phase, wait_ns);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A::COLS) : "memory");
}
#undef FBP_TC_ISSUE

}  // namespace fbp
