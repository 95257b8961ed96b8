// tcgen05 building blocks shared by the tensor-core jet kernels that keep the
// pair-dependent operand in tensor memory: 8-column TMEM loads and stores, an
// MMA with A in TMEM, the TF32 split and the K-major layout of the B operands.
#pragma once

#include "jet.cuh"

namespace fbp {

// The network's compile-time shape without W2 in SParams: the kernels below
// keep it only as B operands.
template <class B>
struct TcCfg : B {
    static constexpr bool W2S = false;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: start, leading (K) and stride (M/N) byte
// offsets between core matrices, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::tf32: FP32 accumulator, TF32 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t umma_idesc_tf32(int M, int N) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait: true when the phase completed, false once limit_ns of wall
// time has passed without it.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t parity, uint64_t limit_ns) {
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(mbar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

constexpr uint64_t TC_WAIT_NS = 200000000ull;  // 0.2 s: an MMA group takes microseconds
constexpr uint64_t TC_TEST_WAIT_NS = 1000000ull;  // 1 ms, with FBP_STATUS_TC_TEST_NO_MMA

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                 "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Waits (bounded) for the phase with one polling lane per warp; false on a time-out.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t mbar, uint32_t parity, uint64_t limit_ns, int lane) {
    int ok = 1;
    if (lane == 0) ok = mbar_wait_bounded(mbar, parity, limit_ns);
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D (TMEM) (+)= A (TMEM, one 32-bit column per K element, row = lane) B^T (shared memory)
__device__ __forceinline__ void umma_tf32_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// v = hi + lo with hi = v rounded to TF32's 10 mantissa bits (ties away), so
// |lo| <= 2^-12 |v|; the MMA reads the top 10 bits of lo, an error of at most
// 2^-22 |v|, of either sign.  (Truncating v instead doubles lo and the error: steps
// 3-4% faster, but the gradients' error against 64 bits 3.2e-7 -> 3.7e-7 for
// 3-32-32-1 networks; cvt.rna.tf32 in place of the two integer operations: 5-10%
// slower.)
__device__ __forceinline__ void split_tf32_rn(float v, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
    lo = v - hi;
}

__device__ __forceinline__ void split2_tf32_rn(float2 v, float2& hi, float2& lo) {
    hi = make_float2(__uint_as_float((__float_as_uint(v.x) + 0x1000u) & 0xFFFFE000u),
                     __uint_as_float((__float_as_uint(v.y) + 0x1000u) & 0xFFFFE000u));
    lo = fma2(hi, dup2(-1.0f), v);
}

// Splits 8 values and stores them as columns [col, col+8) (hi) and
// [col + lo_off, ...) (lo) of this thread's TMEM lane.
__device__ __forceinline__ void tmem_st_split8(uint32_t col, uint32_t lo_off, const float (&v)[8]) {
    float hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float2 a, b;
        split2_tf32_rn(make_float2(v[i], v[i + 1]), a, b);
        hi[i] = a.x, hi[i + 1] = a.y;
        lo[i] = b.x, lo[i + 1] = b.y;
    }
    tmem_st8(col, hi);
    tmem_st8(col + lo_off, lo);
}

// One warp's 16 x 8 x 8 product with TF32 operands and FP32 sums: D = A B
// (ZERO) or D += A B.  Lane (g, t) = (lane / 4, lane % 4) holds A (g, t),
// (g + 8, t), (g, t + 4), (g + 8, t + 4), B (t, g), (t + 4, g) and D (g, 2t),
// (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1).
template <bool ZERO = false>
__device__ __forceinline__ void mma_tf32(float (&d)[4], const float (&a)[4], const float (&b)[2]) {
    if constexpr (ZERO)
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])),
              "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b[0])), "r"(__float_as_uint(b[1])), "f"(0.f));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])),
              "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b[0])), "r"(__float_as_uint(b[1])));
}

// B operand with H K-elements per row in the no-swizzle K-major layout: core
// matrices of 8 rows x 4 floats, 128 bytes apart along K, 32 H bytes along the rows.
template <int H>
struct KMajor {
    static constexpr uint32_t LBO = 128, SBO = 32 * H;
    // float offset of (row, k), and the (row, k) of offset o: a loop over
    // offsets fills the operand without bank conflicts
    __device__ __forceinline__ static int off(int row, int k) {
        return (row >> 3) * 8 * H + (k >> 2) * 32 + (row & 7) * 4 + (k & 3);
    }
    __device__ __forceinline__ static void at(int o, int& row, int& k) {
        row = (o / (8 * H)) * 8 + ((o >> 2) & 7);
        k = ((o % (8 * H)) >> 5) * 4 + (o & 3);
    }
};

// Activations of the tensor-core kernels: from a = sigma and tp = sigma' the
// second and third derivatives are products with the neuron's o (c f(o z)),
//   tanh, adaptive tanh (c o = 1):  tp = 1 - (o a)^2, tpp = -2 o^2 a tp, tppp = o^2 tp (4 - 6 tp)
//   sin, adaptive sin:              tpp = -o^2 a,     tppp = -o^2 tp
// so the tpp operand of an MMA is m2 = a tp (tanh) or a itself (sin), with
// k2 = tpp / m2 in the other operand.
template <class C>
struct TcAct {
    // L2: layer 2 (else layer 1)
    template <bool L2>
    static constexpr int ACT = L2 ? act_layer2(C::ACT) : act_layer1(C::ACT);
    template <bool L2>
    static constexpr bool SIN = ACT<L2> == FBP_ACT_SIN || ACT<L2> == FBP_ACT_ADAPTIVE_SIN;
    // k2 and o^2 of a neuron with activation parameter o
    template <bool L2>
    __device__ __forceinline__ static float k2(float o) {
        return (SIN<L2> ? -1.0f : -2.0f) * (C::EXTRA > 0 ? o * o : 1.0f);
    }
    // neurons n, n + 1 at the pre-activations z: value and first derivative
    template <bool L2>
    __device__ __forceinline__ static void first(const SParams<C>& S, int n, float2 z, float2& a, float2& tp) {
        if constexpr (ACT<L2> == FBP_ACT_TANH) {
            a = tanh_fast2(z);
            tp = fma2(make_float2(-a.x, -a.y), a, dup2(1.0f));
        } else if constexpr (SIN<L2>) {
            const float2 c = make_float2(act_c<C, L2>(S, n), act_c<C, L2>(S, n + 1));
            const float2 o = make_float2(act_o<C, L2>(S, n), act_o<C, L2>(S, n + 1));
            float2 sn, cs;
            sincos2(C::EXTRA > 0 ? mul2(o, z) : z, sn, cs);
            a = C::EXTRA > 0 ? mul2(c, sn) : sn;
            tp = C::EXTRA > 0 ? mul2(mul2(c, o), cs) : cs;
        } else {
            using A = Act<ACT<L2>>;
            float d2, d3;
            A::derivs(A::stored(z.x, act_o<C, L2>(S, n)), act_c<C, L2>(S, n), act_o<C, L2>(S, n), a.x, tp.x, d2, d3);
            A::derivs(A::stored(z.y, act_o<C, L2>(S, n + 1)), act_c<C, L2>(S, n + 1), act_o<C, L2>(S, n + 1), a.y, tp.y,
                      d2, d3);
        }
    }
    template <bool L2>
    __device__ __forceinline__ static float2 m2(float2 a, float2 tp) {
        return SIN<L2> ? a : mul2(a, tp);
    }
    template <bool L2>
    __device__ __forceinline__ static float2 oo(const SParams<C>& S, int n) {
        const float2 o = make_float2(act_o<C, L2>(S, n), act_o<C, L2>(S, n + 1));
        return mul2(o, o);
    }
    // the second derivative from m2 of neurons n, n + 1, the third from tp
    template <bool L2>
    __device__ __forceinline__ static float2 second(const SParams<C>& S, int n, float2 m2) {
        const float2 t = mul2(dup2(SIN<L2> ? -1.0f : -2.0f), m2);
        return C::EXTRA > 0 ? mul2(oo<L2>(S, n), t) : t;
    }
    template <bool L2>
    __device__ __forceinline__ static float2 third(const SParams<C>& S, int n, float2 tp) {
        const float2 t = SIN<L2> ? make_float2(-tp.x, -tp.y) : mul2(tp, fma2(dup2(-6.0f), tp, dup2(4.0f)));
        return C::EXTRA > 0 ? mul2(oo<L2>(S, n), t) : t;
    }
};

}  // namespace fbp
