// Quantized weights on mma.sync (the streaming matvec, the small-batch matmul and the one-launch step): two codes to two f16 in two
// instructions; and the GeGLU epilogue of every kernel that has one.
#pragma once
#include "tcgen05_util.cuh"

namespace {

// gelu_tanh(gate) * up with gate and up rounded to f16 first, as the separate projections would store them, and the
// element-wise kernel's arithmetic (shaders/gelu.metal:23-37)
__device__ __forceinline__ float geglu_f(float gate, float up) {
    const float x = __half2float(__float2half_rn(gate)), u = __half2float(__float2half_rn(up));
    float inner = 0.7978845608f * (x + 0.044715f * (x * x * x));
    inner = fminf(fmaxf(inner, -10.0f), 10.0f);
    return 0.5f * x * (1.0f + tanhf(inner)) * u;
}
// two codes, BITS wide at bit BITS * l of each half of w, as f16 (q - Z) 2^-9: in place they are the f16 subnormals
// q 2^(BITS l - 24), which one multiply-add moves to the common scale, exactly
template <int BITS, int Z>
__device__ __forceinline__ uint32_t codes_f16(uint32_t w, int l) {
    constexpr uint32_t one = (1u << BITS) - 1u;
    const uint32_t v = w & ((one | one << 16) << (BITS * l));      // q 2^(BITS l - 24)
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&v), __float2half2_rn((float)(1 << (15 - BITS * l))),
                              __float2half2_rn(-(float)Z / 512.0f));
    return *reinterpret_cast<const uint32_t *>(&r);
}

}  // namespace
