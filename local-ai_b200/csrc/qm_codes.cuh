// Quantized weights on mma.sync at few batch rows (qmatmul_sm.cu; step_small.cu): code words from shared memory, two codes to two
// f16 in two instructions, the MMA, and the GeGLU epilogue.
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
// (Neither the MMA nor the loads are volatile: the compiler overlaps the steps of an unrolled loop.)
__device__ __forceinline__ void sm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// N consecutive 32-bit words at byte `at` (even) of a 4-byte aligned array in shared memory, the bytes of each in the order 0, 2, 1, 3: a
// mask then pairs neighbouring codes in the halves of a register.
template <int N>
__device__ __forceinline__ void lds_codes(const uint8_t *smem, uint32_t at, uint32_t (&w)[N]) {
    const uint32_t sel = (at & 2u) ? 0x5342u : 0x3120u;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(smem + (at & ~3u));
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; i++) r[i] = src[i];
#pragma unroll
    for (int i = 0; i < N; i++) w[i] = __byte_perm(r[i], r[i + 1], sel);
}
__device__ __forceinline__ uint32_t lds16(const uint8_t *smem, uint32_t at) { return *reinterpret_cast<const uint16_t *>(smem + at); }

// two codes, BITS wide at bit BITS * l of each half of w, as f16 (q - Z) 2^-9
template <int BITS, int Z>
__device__ __forceinline__ uint32_t codes_f16(uint32_t w, int l) {
    constexpr uint32_t one = (1u << BITS) - 1u;
    const uint32_t v = w & ((one | one << 16) << (BITS * l));      // q 2^(BITS l - 24)
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&v), __float2half2_rn((float)(1 << (15 - BITS * l))),
                              __float2half2_rn(-(float)Z / 512.0f));
    return *reinterpret_cast<const uint32_t *>(&r);
}

}  // namespace
