// Attention over TurboQuant codes with the sixteen warps of a CTA side by side on one block of 64 keys and 8 q-heads.
//
// In attention_tq_mma.cu a warp owns 32 keys and all head_dim dims: a tile is one long chain (about 4500 cycles the first time round)
// and the warps' accumulators are merged at the end (another 2200).  That suits long runs of keys.  Here warp w owns the
// head_dim / 8 dims of part w mod 8 and half w / 8 of the block's keys, in both contractions, so a block is short (2600 cycles) and
// there is little to merge; the price is three barriers per block, around the exchange of the logits.  Operands, table and
// precision are those of that file:
//   * S^T[64 keys x 8 heads]: part w contracts over dims HD/8 w .. + HD/8 - 1, thread (g, t) with the HD/32 dims at HD/8 w + HD/32 t of
//     keys 16 mt + g, + 8 (the code words of a warp lie side by side: no bank conflicts at a row stride of CB + 16);
//   * thread (head = tid & 7, key tid >> 3) adds the eight parts, scales by the key norm and takes part in the softmax of its head;
//   * O^T[HD/8 dims x 8 heads] of part w += V^T . P: thread (g, t) decodes dims HD/8 w + HD/64 g .. of keys 2t, 2t+1, 2t+8, 2t+9.
#pragma once
#include "attention_tq_tile.cuh"

namespace {

template <typename C>
struct Wide {
    static constexpr int HD = C::HD, BITS = C::BITS, CB = C::CB, FB = C::FB;
    static constexpr int NW = 16, NT = NW * 32, KB = 64, MT = KB / 32;   // keys of a block, 16-key tiles of a warp
    static constexpr int RS = CB + 16, STAGE = 2 * KB * RS;    // K rows, then V rows
    static constexpr int KS = HD / 128, TL = HD / 128;         // k16 steps of QK and 16-row tiles of PV of a warp
    static constexpr int PS = KB + 8;                          // row (head) of P, halves
    static constexpr int PART_BYTES = 8 * KB * G * 4, P_BYTES = G * PS * 2 * (C::HILO ? 2 : 1);
    static constexpr int SCRATCH = PART_BYTES + P_BYTES + NW * G * 4 + 4 * KB * 4;   // parts, P, maxima, norms of two blocks
};
// NB bits at bit `bit` of a shared-memory row (rows are 16-byte aligned; a multiple of NB when NB divides 32)
template <int NB>
__device__ __forceinline__ uint32_t row_bits(const uint8_t *row, uint32_t bit) {
    if constexpr (NB == 8) return row[bit >> 3];
    else if constexpr (NB == 16) return *reinterpret_cast<const uint16_t *>(row + (bit >> 3));
    else {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(row) + (bit >> 5);
        if constexpr (32 % NB == 0) return w[0] >> (bit & 31u);
        else return __funnelshift_r(w[0], w[1], bit);   // (the 16 bytes after a row are there)
    }
}
template <int FB, int I>
__device__ __forceinline__ uint2 table_entry(const uint2 *lut_lane, uint32_t v) {
    return lut_lane[((v >> (I * FB)) & ((1u << FB) - 1u)) * LUT_COPIES];
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {   // (free to move)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The CTA's sixteen working warps (it may have others).
__device__ __forceinline__ void wide_sync() { asm volatile("barrier.cta.sync.aligned 1, 512;\n" ::: "memory"); }
__device__ __forceinline__ bool wide_sync_or(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred.aligned q, 1, 512, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"((uint32_t)v)
        : "memory");
    return r != 0;
}

template <typename C>
struct WideAcc {
    float o[Wide<C>::TL][4];   // dims HD/8 warp + HD/64 g + 2 tile (+ 1: elements 2, 3) of heads 2t, 2t + 1
    float m, l;                // head tid & 7: running maximum, this thread's part of the sum (o: of this half of the keys)
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < Wide<C>::TL; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
        m = -INFINITY;
        l = 0.f;
    }
};
// One block: its codes at `stage` and norms (times gamma; K's, then V's) at `norms` are in shared memory and behind a barrier; n >= 1
// keys count.  q: this lane's query fragments {hi01, hi23, lo01, lo23} of its HD/32 dims.  Ends without a barrier; the caller has
// one before the next block.
template <typename C>
__device__ __forceinline__ void wide_block(WideAcc<C> &acc, const uint8_t *stage, const float *norms, int n, const uint4 (&q)[Wide<C>::KS],
                                           const uint2 *lut_lane, uint8_t *scratch, int tid) {
    using W = Wide<C>;
    constexpr int MT = W::MT, KS = W::KS, TL = W::TL, FB = C::FB, BITS = C::BITS, HD = C::HD;
    const int lane = tid & 31, warp = tid >> 5, dw = warp & 7, mt0 = (warp >> 3) * MT, g = lane >> 2, t = lane & 3;
    float *part = reinterpret_cast<float *>(scratch);                                  // [warp][key][head]
    __half *ps = reinterpret_cast<__half *>(scratch + W::PART_BYTES);                  // [head][key] (HILO: twice)
    float *wmax = reinterpret_cast<float *>(scratch + W::PART_BYTES + W::P_BYTES);     // [warp][head]

    // ---- this warp's part of S^T ----
    {
        constexpr int NB = HD / 32 * BITS, KF = C::HILO ? 2 : 1;   // bits of a thread's dims; table fields per k-step
        const uint8_t *k0 = stage + (mt0 * 16 + g) * W::RS;
        const uint32_t bit = (uint32_t)(dw * (HD / 8) + t * (HD / 32)) * BITS;
#pragma unroll 1
        for (int mt = 0; mt < MT; mt++) {   // (rolled: short code is fetched faster than this runs)
            uint32_t v[2][(NB + 31) / 32];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint8_t *row = k0 + (mt * 16 + h * 8) * W::RS;
                if constexpr (NB <= 32) {
                    v[h][0] = row_bits<NB>(row, bit);
                } else {
                    v[h][0] = row_bits<24>(row, bit);          // (48 or 64 bits: two pieces of whole fields)
                    v[h][1] = row_bits<24>(row, bit + NB / 2);
                    if constexpr (NB == 64) {
                        v[h][0] = reinterpret_cast<const uint32_t *>(row)[bit >> 5];
                        v[h][1] = reinterpret_cast<const uint32_t *>(row)[(bit >> 5) + 1];
                    }
                }
            }
            float c[2][4] = {};   // high and low query parts
            static_for<KS>([&](auto S) {
                constexpr int s = decltype(S)::value;
                constexpr int word = NB <= 32 ? 0 : s / (KS / 2), f = NB <= 32 ? s * KF : (s % (KS / 2)) * KF;
                if constexpr (!C::HILO) {
                    const uint2 x = table_entry<FB, f>(lut_lane, v[0][word]), y = table_entry<FB, f>(lut_lane, v[1][word]);
                    const uint32_t a[4] = {x.x, y.x, x.y, y.y};
                    mma_f16(c[0], a, q[s].x, q[s].y);
                    mma_f16(c[1], a, q[s].z, q[s].w);
                } else {
                    const uint2 x0 = table_entry<FB, f>(lut_lane, v[0][word]), x1 = table_entry<FB, f + 1>(lut_lane, v[0][word]);
                    const uint2 y0 = table_entry<FB, f>(lut_lane, v[1][word]), y1 = table_entry<FB, f + 1>(lut_lane, v[1][word]);
                    const uint32_t ah[4] = {x0.x, y0.x, x1.x, y1.x}, al[4] = {x0.y, y0.y, x1.y, y1.y};
                    mma_f16(c[0], ah, q[s].x, q[s].y);
                    mma_f16(c[1], ah, q[s].z, q[s].w);
                    mma_f16(c[1], al, q[s].x, q[s].y);
                }
            });
            float *dst = part + (dw * W::KB + (mt0 + mt) * 16 + g) * G + 2 * t;
            *reinterpret_cast<float2 *>(dst) = make_float2(c[0][0] + c[1][0], c[0][1] + c[1][1]);
            *reinterpret_cast<float2 *>(dst + 8 * G) = make_float2(c[0][2] + c[1][2], c[0][3] + c[1][3]);
        }
    }
    wide_sync();
    // ---- softmax: head tid & 7, key tid >> 3 ----
    const int head = tid & 7, key = tid >> 3;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) s += part[w * W::KB * G + tid];
    s = key < n ? s * norms[key] : -INFINITY;
    float mx = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    if (lane < G) wmax[warp * G + lane] = mx;
    wide_sync();
    float m_new = acc.m;
#pragma unroll
    for (int w = 0; w < W::NW; w++) m_new = fmaxf(m_new, wmax[w * G + head]);
    const float resc = soft_exp<C::HILO>(acc.m - m_new);   // (m_new is finite: n >= 1)
    acc.m = m_new;
    const float p = soft_exp<C::HILO>(s - m_new), pv = p * norms[W::KB + key];
    acc.l = acc.l * resc + p;
    const __half hi = __float2half_rn(pv);
    ps[head * W::PS + key] = hi;
    if constexpr (C::HILO) ps[(G + head) * W::PS + key] = __float2half_rn(pv - __half2float(hi));
    if (__any_sync(0xffffffffu, resc != 1.0f)) {
        const float r0 = __shfl_sync(0xffffffffu, resc, 2 * t), r1 = __shfl_sync(0xffffffffu, resc, 2 * t + 1);   // (lane h < 8 has head h)
#pragma unroll
        for (int i = 0; i < TL; i++) {
            acc.o[i][0] *= r0; acc.o[i][1] *= r1; acc.o[i][2] *= r0; acc.o[i][3] *= r1;
        }
    }
    wide_sync();
    // ---- O^T += V^T . P ----
    {
        constexpr int NB = HD / 64 * BITS;
        const uint8_t *v0 = stage + (W::KB + mt0 * 16 + 2 * t) * W::RS;
        const uint32_t bit = (uint32_t)(dw * (HD / 8) + g * (HD / 64)) * BITS;
#pragma unroll 1
        for (int mt = 0; mt < MT; mt++) {   // (rolled: short code is fetched faster than this runs)
            uint32_t v[4];   // keys 2t, 2t + 1, 2t + 8, 2t + 9 of this tile
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = row_bits<NB>(v0 + (16 * mt + (i & 1) + 8 * (i >> 1)) * W::RS, bit);
            const uint32_t *pw = reinterpret_cast<const uint32_t *>(ps + g * W::PS) + 8 * (mt0 + mt) + t;
            const uint32_t b0 = pw[0], b1 = pw[4];
            uint32_t l0 = 0, l1 = 0;
            if constexpr (C::HILO) {
                l0 = pw[G * W::PS / 2];
                l1 = pw[G * W::PS / 2 + 4];
            }
            static_for<(C::HILO ? TL : TL / 2)>([&](auto U) {   // a table field: four dims (two tiles), or two dims in two parts
                constexpr int u = decltype(U)::value;
                const uint2 e0 = table_entry<FB, u>(lut_lane, v[0]), e1 = table_entry<FB, u>(lut_lane, v[1]);
                const uint2 e2 = table_entry<FB, u>(lut_lane, v[2]), e3 = table_entry<FB, u>(lut_lane, v[3]);
                const uint32_t ax[4] = {__byte_perm(e0.x, e1.x, 0x5410), __byte_perm(e0.x, e1.x, 0x7632), __byte_perm(e2.x, e3.x, 0x5410),
                                        __byte_perm(e2.x, e3.x, 0x7632)};
                const uint32_t ay[4] = {__byte_perm(e0.y, e1.y, 0x5410), __byte_perm(e0.y, e1.y, 0x7632), __byte_perm(e2.y, e3.y, 0x5410),
                                        __byte_perm(e2.y, e3.y, 0x7632)};
                if constexpr (!C::HILO) {
                    mma_f16(acc.o[2 * u], ax, b0, b1);
                    mma_f16(acc.o[2 * u + 1], ay, b0, b1);
                } else {
                    mma_f16(acc.o[u], ax, b0, b1);
                    mma_f16(acc.o[u], ax, l0, l1);
                    mma_f16(acc.o[u], ay, b0, b1);
                }
            });
        }
    }
}

}  // namespace
