// Shared helpers of libfbpgpu: status handling, launch checks, jet layout.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/fbpgpu.h"

namespace fbp {

// Thread-local message for fbp_last_error().
void set_error(const char* fmt, ...);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

#define FBP_REQUIRE(cond, code, ...)      \
    do {                                  \
        if (!(cond)) {                    \
            ::fbp::set_error(__VA_ARGS__); \
            return (code);                \
        }                                 \
    } while (0)

#define FBP_CUDA_CHECK(expr)                                                           \
    do {                                                                               \
        cudaError_t e_ = (expr);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            ::fbp::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), \
                             __FILE__, __LINE__);                                      \
            return FBP_ERR_CUDA;                                                       \
        }                                                                              \
    } while (0)

#define FBP_LAUNCH_CHECK() FBP_CUDA_CHECK(cudaGetLastError())

constexpr int kSM = 152;  // GB300 SM count (grid sizing hint; queried at run time too)

// Elements per tile of the exclusive int32 scan (takes.cu): its scratch holds
// one sum per tile plus the total.
constexpr int kScanTile = 2048;

// Per-device caches (kernel attributes, occupancy-sized grids) are indexed by
// the current device, 0 .. FBP_MAX_DEVICES - 1.
constexpr int FBP_MAX_DEVICES = 64;
int current_device();
int sm_count();

__host__ __device__ constexpr int popc_const(int v) {
    return v == 0 ? 0 : (v & 1) + popc_const(v >> 1);
}

// Second-derivative part of a jet, from the d2mask: bits 0-2 name the dims
// whose pure second derivatives are needed.  The dims of the group (all of
// them with FBP_D2_LAPLACIAN, bit 3; else the dims named by bits 4-6, see
// FBP_D2_GROUP) share one slot that holds the sum of their second
// derivatives (a Laplacian, propagated directly as in the forward-Laplacian
// scheme); every other masked dim has a slot of its own.  Slot order: the
// group's slot first, then the single dims ascending.
__host__ __device__ constexpr int d2_group(int d2) {
    return (d2 & FBP_D2_LAPLACIAN) ? (d2 & 7) : ((d2 >> 4) & 7 & d2);
}
__host__ __device__ constexpr int d2_singles(int d2) { return d2 & 7 & ~d2_group(d2); }
__host__ __device__ constexpr bool d2_lap(int d2) { return d2_group(d2) != 0; }
__host__ __device__ constexpr int d2_slots(int d2) { return (d2_group(d2) ? 1 : 0) + popc_const(d2_singles(d2)); }

// Jet layout: [u, d/dx_0..d/dx_{XD-1}, then the second-derivative slots: one
// per bit i of the d2mask ascending, or the single Laplacian slot].
__host__ __device__ constexpr int jet_size(int xd, int d2) { return 1 + xd + d2_slots(d2); }

// Index of the s-th set bit of mask among bits 0..7 (0 when there is none).
__host__ __device__ constexpr int nth_bit(int mask, int s) {
    int c = 0;
    for (int d = 0; d < 8; ++d)
        if ((mask >> d) & 1) {
            if (c == s) return d;
            ++c;
        }
    return 0;
}

// Row stride (floats) of the per-pair and per-slot jet records [first J | second J]:
// 2J rounded up to a multiple of 4 so that rows can be moved as float4.
__host__ __device__ constexpr int rec_stride(int J) { return (2 * J + 3) / 4 * 4; }

// Compile-time table of the set bits of a mask (up to 3): DimsOf<M>::get(s) is
// the s-th set bit, folded to a constant when s is a constant.
template <int M>
struct DimsOf {
    static constexpr int d0 = nth_bit(M, 0), d1 = nth_bit(M, 1), d2 = nth_bit(M, 2);
    __host__ __device__ static constexpr int get(int s) { return s == 0 ? d0 : (s == 1 ? d1 : d2); }
};

// Dims whose pure second derivatives second-derivative slot s of a d2mask sums
// (the group for the group's slot, else one dim).
template <int D2>
__host__ __device__ constexpr int d2_slot_dims(int s) {
    return d2_group(D2) ? (s == 0 ? d2_group(D2) : (1 << DimsOf<d2_singles(D2)>::get(s - 1)))
                        : (1 << DimsOf<D2 & 7>::get(s));
}

// 2^x and 1 / x by the hardware's approximations, denormals flushed to zero.
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// tanh from the identity tanh|x| = (1 - e) / (1 + e), e = exp(-2|x|), with the
// hardware's exponential and reciprocal and the sign restored.  e lies in
// [0, 1], so nothing overflows, and where the instructions flush (e below
// 2^-126, |x| below 2^-127) 1 - e and 1 + e are unchanged; the forms that keep
// denormals (__expf, __fdividef) take about twice the instructions.  The
// absolute error is about 1e-7 over the whole line (checked against torch.tanh
// by tests/test_gpu_step.py::test_fast_tanh_error).
constexpr float kTanhScale = -2.8853900817779268f;  // -2 log2(e)
__device__ __forceinline__ float tanh_fast(float x) {
    const float e = ex2_ftz(fabsf(x) * kTanhScale);
    return copysignf((1.0f - e) * rcp_ftz(1.0f + e), x);
}

// One parameter's Adam step (optax.adam: moments, bias corrections bc1 = 1 - b1^t,
// bc2 = 1 - b2^t, scale(-lr)).
__device__ __forceinline__ void adam_element(float& theta, float& m1, float& m2, float g, float lr, float b1, float b2,
                                             float eps, float eps_root, float bc1, float bc2) {
    const float mu = (1.0f - b1) * g + b1 * m1;
    const float nu = (1.0f - b2) * g * g + b2 * m2;
    m1 = mu;
    m2 = nu;
    const float mh = mu / bc1;
    const float nh = nu / bc2;
    theta = theta + (-lr) * (mh / (sqrtf(nh + eps_root) + eps));
}

// Programmatic dependent launch between the kernels of a step: the next kernel
// may be set up while the one before it ends, and waits, before it touches
// global memory, until that one has completed and its writes are visible.  It
// does nothing for kernels launched without it.  (No kernel lets the next one
// start early: waiting CTAs then hold registers and tensor memory that the list
// kernels on the other stream could use -- a step of 16381 redrawn points 118
// -> 132 us, Burgers 67 -> 72.)  The forward is launched without it, and under
// the dynamic schedule the adjoint follows the memset of its item counter, so
// neither overlaps the end of a kernel.  The 1D oscillator's step 35.0 -> 33.0 us.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel that begins with pdl_wait, so that its launch overlaps the
// end of the kernel before it on the stream.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

inline int jet_size_rt(int xd, int d2) { return 1 + xd + d2_slots(d2); }

}  // namespace fbp
