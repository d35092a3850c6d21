// Rows of the KV cache and of the query held by a warp (turboquant.cu; step_small.cu runs the same arithmetic inside the decode
// step): head norm, rotary embedding, the codec's rotation and codes, the attention kernels' query fragments.
#pragma once
#include <cuda_fp16.h>
#include <math.h>
#include <stdint.h>

namespace {

// Rotates x (HD / 32 consecutive dims per lane): Walsh-Hadamard butterflies in ascending stride, lower = a + b, upper = a - b.
template <int DPL>
__device__ __forceinline__ void fwht_warp_row(float (&x)[DPL], int lane) {
#pragma unroll
    for (int len = 1; len < DPL; len <<= 1)
#pragma unroll
        for (int i = 0; i < DPL; i++)
            if (!(i & len)) {
                const float a = x[i], b = x[i + len];
                x[i] = __fadd_rn(a, b);
                x[i + len] = __fsub_rn(a, b);
            }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const bool upper = lane & m;
#pragma unroll
        for (int i = 0; i < DPL; i++) {
            const float o = __shfl_xor_sync(0xffffffffu, x[i], m);
            x[i] = upper ? __fsub_rn(o, x[i]) : __fadd_rn(x[i], o);
        }
    }
}
// The codes (this lane's HD / 32, LSB first) of one row held by a warp, HD / 32 consecutive dims per lane, whose norm is known
// (TurboQuant::encode_into).
template <int HD, int BITS>
__device__ __forceinline__ unsigned long long encode_warp_row(float (&x)[HD / 32], float norm, const float (&lv)[1 << BITS],
                                                              const float (&sg)[HD / 32], int lane) {
    constexpr int DPL = HD / 32, NLEV = 1 << BITS;
    const float inv = norm > 0.f ? __fdiv_rn(1.0f, norm) : 0.f;
#pragma unroll
    for (int i = 0; i < DPL; i++) x[i] = __fmul_rn(norm > 0.f ? __fmul_rn(x[i], inv) : x[i], sg[i]);
    fwht_warp_row<DPL>(x, lane);
    const float inv_sqrt_d = __fdiv_rn(1.0f, __fsqrt_rn((float)HD));
    unsigned long long word = 0;
#pragma unroll
    for (int i = 0; i < DPL; i++) {
        const float v = __fmul_rn(x[i], inv_sqrt_d);
        unsigned best = 0;
        float bd = INFINITY;
#pragma unroll
        for (int j = 0; j < NLEV; j++) {
            const float dd = fabsf(__fsub_rn(v, lv[j]));
            if (dd < bd) { bd = dd; best = (unsigned)j; }
        }
        word |= (unsigned long long)best << (BITS * i);
    }
    return word;
}
// The codes of a row where encode_warp_row left them, to any memory.
template <int HD, int BITS>
__device__ __forceinline__ void store_warp_codes(unsigned long long word, int lane, uint8_t *dst) {
    constexpr int LB = HD / 32 * BITS;   // bits of one lane: 8 .. 64, or 12 (tq3 at head_dim 128)
    if constexpr (LB == 12) {            // two lanes share three bytes
        const unsigned w = (unsigned)word | (__shfl_down_sync(0xffffffffu, (unsigned)word, 1) << 12);
        if (!(lane & 1)) {
            dst += (lane >> 1) * 3;
            dst[0] = (uint8_t)w;
            dst[1] = (uint8_t)(w >> 8);
            dst[2] = (uint8_t)(w >> 16);
        }
    } else {
        dst += lane * (LB / 8);
#pragma unroll
        for (int i = 0; i < LB / 8; i++) dst[i] = (uint8_t)(word >> (8 * i));
    }
}
// x = f16(x / rms * w) for a head of 256 dims, eight consecutive ones per lane.  Mean square: 32-dim groups as shuffle trees
// (strides 16, 8 across lanes; 4, 2, 1 inside), then the groups in order.
__device__ __forceinline__ void warp_head_norm(float (&x)[8], const float (&w)[8], float eps) {
    float tot = 0.f, s[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        s[e] = x[e] * x[e];
        s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
        s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int e = 0; e < o; e++) s[e] += s[e + o];
#pragma unroll
    for (int g = 0; g < 8; g++) tot += __shfl_sync(0xffffffffu, s[0], 4 * g);
    const float rms = rsqrtf(tot / 256.0f + eps);
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = __half2float(__float2half_rn(x[e] * rms * w[e]));
}
// Rotates dims d and d + 128 (d < angles) of such a head; cs, sn belong to dim (8 lane + e) mod 128.
__device__ __forceinline__ void warp_rope(float (&x)[8], const float (&cs)[8], const float (&sn)[8], unsigned angles, int lane) {
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const float other = __shfl_xor_sync(0xffffffffu, x[e], 16);
        const bool low = lane < 16;
        const float x0 = low ? x[e] : other, x1 = low ? other : x[e];
        const float v = low ? x0 * cs[e] - x1 * sn[e] : x0 * sn[e] + x1 * cs[e];
        if (((unsigned)(8 * lane + e) & 127u) < angles) x[e] = __half2float(__float2half_rn(v));
    }
}
// The tensor-core attention kernel's first steps on a query head: sign, transform, scale, an f16 and the f16 of the remainder.
// f[0], f[1]: the fragments of dims 8 lane + 0 .. 3 and + 4 .. 7, entries 2 (lane & 7) and the next (TqAttnParams::qfrag).
__device__ __forceinline__ void warp_query_frag(float (&x)[8], const float (&sg)[8], float q_scale, int lane, uint4 (&f)[2]) {
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = __fmul_rn(x[e], sg[e]);
    fwht_warp_row<8>(x, lane);
    const float k = __fdiv_rn(q_scale, __fsqrt_rn(256.0f));
    unsigned hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float v0 = __fmul_rn(x[2 * i], k), v1 = __fmul_rn(x[2 * i + 1], k);
        const __half2 a = __floats2half2_rn(v0, v1);
        const __half2 b = __floats2half2_rn(__fsub_rn(v0, __low2float(a)), __fsub_rn(v1, __high2float(a)));
        hi[i] = *reinterpret_cast<const unsigned *>(&a);
        lo[i] = *reinterpret_cast<const unsigned *>(&b);
    }
    f[0] = make_uint4(hi[0], hi[1], lo[0], lo[1]);
    f[1] = make_uint4(hi[2], hi[3], lo[2], lo[3]);
}
// The reference's sequential f32 sum of a row of squares, in index order, and its root.
template <int HD>
__device__ __forceinline__ float sequential_norm(const float *sq) {
    const float4 *r4 = reinterpret_cast<const float4 *>(sq);
    float s = 0.f;
#pragma unroll 8
    for (int i = 0; i < HD / 4; i++) {
        const float4 a = r4[i];
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
    }
    return __fsqrt_rn(s);
}

}  // namespace
