// What the kernels that attend over TurboQuant codes on mma.sync share: the configuration, the table of levels and one warp's
// step over a tile of keys (attention_tq_mma.cu explains the arithmetic; step_small.cu runs the same step inside the decode step).
#pragma once
#include <utility>

#include "attention_tq.h"
#include "tcgen05_util.cuh"

namespace {

constexpr int G = 8;             // q-heads per CTA (MMA N)
constexpr int LUT_COPIES = 16;   // an 8-byte shared load is served per half-warp, so 16 copies are conflict-free

template <int HD_, int BITS_>
struct AttnCfg {
    static constexpr int HD = HD_, BITS = BITS_;
    static constexpr int CB = HD * BITS / 8;            // code bytes per row
    static constexpr bool HILO = BITS > 2 || HD != 256; // levels and P as an f16 and the f16 of the remainder
    static constexpr int FB = HILO ? 2 * BITS : 8;      // table index bits
    static constexpr int NENT = 1 << FB;
    static constexpr int MT = HD == 512 ? 1 : 2;        // 16-key MMA tiles per warp step
    static constexpr int KT = 16 * MT;
    static constexpr int NW = 8, NT = NW * 32;
    static constexpr int NS = HD / 16;                  // k16 steps of QK, 16-dim tiles of PV
    static constexpr int DPL = HD / 32;                 // dims per lane where a warp owns a head
    static constexpr bool PAIRS = HD <= 256;            // V lookups serve two keys at once (attn_tile); at 512 dims two parts of them leave no registers
    static constexpr int NO = HILO && PAIRS ? 2 * NS : NS;   // accumulator tiles of a warp
    static constexpr bool QSMEM = NO > 16;              // query fragments stay in shared memory (registers hold the accumulators)
    // Row strides in the ring: chosen so that the fragment reads spread over the banks.
    static constexpr int KRS = (BITS == 2 && HD == 256) ? CB : CB + 16;
    static constexpr int VRS = CB + 16;
    static constexpr int STAGE = KT * (KRS + VRS);
    static constexpr int LUT_BYTES = NENT * LUT_COPIES * 8;
    static constexpr int Q_BYTES = NS * 32 * 16;        // query: f32 [NS][32][4], then the packed fragments in place
    static constexpr int ACC_BYTES = NW * NS * 4 * 32 * 4;   // merge staging, reuses query and ring memory
    static constexpr int RING_OFF = LUT_BYTES + Q_BYTES;
    // Merged rows (a head of one split): four floats of padding after every HD / 8 dims (their writers' lanes are HD / 8 dims
    // apart).  A CTA of a cluster of n receives n rows for each of its ceil(8 / n) heads, at most 14.
    static constexpr int CPS = HD + 40, ROWS = 14;
    static constexpr int TAIL_BYTES = (2 * NW * G + 2 * ROWS) * 4 + ROWS * CPS * 4;  // (max, sum) of warps and rows, the rows
    static __device__ __forceinline__ int cp_index(int row, int d) { return row * CPS + d + 4 * (d / (HD / 8)); }
    static constexpr int RING_ROOM = 222 * 1024 - TAIL_BYTES - RING_OFF;
    static constexpr int DEPTH_FIT = RING_ROOM / (NW * STAGE);
    static constexpr int DEPTH = DEPTH_FIT > 4 ? 4 : DEPTH_FIT;   // ring slots per warp (DEPTH - 1 tiles in flight)
    static constexpr int SMEM0 = RING_OFF + NW * DEPTH * STAGE;
    static constexpr int TAIL_OFF = SMEM0 > LUT_BYTES + ACC_BYTES ? SMEM0 : LUT_BYTES + ACC_BYTES;
    static constexpr int SMEM = TAIL_OFF + TAIL_BYTES;
    static_assert(DEPTH >= 2, "the ring needs two slots");
    static_assert(SMEM <= 224 * 1024, "shared memory, with room for the static part");
};

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
// the same place in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(addr), "r"(rank));
    return ra;
}
__device__ __forceinline__ void st_cluster_f2(uint32_t a, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
// N 32-bit words of shared memory at an address aligned for the widest load that divides N
template <int N>
__device__ __forceinline__ void lds_words(uint32_t a, uint32_t (&w)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]) : "r"(a + 4 * i));
    } else if constexpr (N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 2)
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(w[i]), "=r"(w[i + 1]) : "r"(a + 4 * i));
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w[i]) : "r"(a + 4 * i));
    }
}
// f(integral_constant<0>) .. f(integral_constant<N - 1>)
template <typename F, int... I>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F &&f) {
    static_for_impl(f, std::make_integer_sequence<int, N>{});
}
// Table address of the FB-bit field at bit O of a word run: lane base + index * 128 bytes.  The multiply-add goes to the
// multiply pipe, which is idle here; the ALU pipe is the busy one.
template <int FB, int O, int N>
__device__ __forceinline__ uint32_t field_addr(const uint32_t (&w)[N], uint32_t lane_base) {
    constexpr int i = O / 32, o = O % 32;
    uint32_t idx, r;
    if constexpr (FB == 8) idx = __byte_perm(w[i], 0u, 0x4440 + o / 8);
    else if constexpr (o + FB > 32) idx = __funnelshift_r(w[i], w[i + 1 < N ? i + 1 : i], o) & ((1u << FB) - 1u);
    else idx = (w[i] >> o) & ((1u << FB) - 1u);
    asm("mad.lo.u32 %0, %1, %2, %3;\n" : "=r"(r) : "r"(idx), "n"(LUT_COPIES * 8), "r"(lane_base));
    return r;
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ uint32_t pack_h2(float x, float y) {
    __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ float2 unpack_h2(uint32_t u) { return __half22float2(*reinterpret_cast<__half2 *>(&u)); }
// f16 of the two values and f16 of what the rounding left
__device__ __forceinline__ void split_h2(float x, float y, uint32_t &hi, uint32_t &lo) {
    hi = pack_h2(x, y);
    const float2 h = unpack_h2(hi);
    lo = pack_h2(x - h.x, y - h.y);
}
template <bool HILO>
__device__ __forceinline__ float soft_exp(float x) {
    return HILO ? expf(x) : __expf(x);
}

// Walsh-Hadamard butterflies over 32 * DPL values held DPL per lane (lane owns consecutive dims), ascending stride.
template <int DPL>
__device__ __forceinline__ void warp_fwht(float (&x)[DPL], int lane) {
#pragma unroll
    for (int len = 1; len < DPL; len <<= 1) {
#pragma unroll
        for (int i = 0; i < DPL; i++) {
            if (!(i & len)) {
                const float a = x[i], b2 = x[i + len];
                x[i] = a + b2;
                x[i + len] = a - b2;
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const bool upper = lane & m;
#pragma unroll
        for (int i = 0; i < DPL; i++) {
            const float o2 = __shfl_xor_sync(0xffffffffu, x[i], m);
            x[i] = upper ? o2 - x[i] : x[i] + o2;
        }
    }
}

// The table of levels at the start of shared memory and gamma, by the whole CTA of NW warps; the levels are a constant operand.  The table is
// complete for all threads after the caller's next barrier.  A thread writes the copies of its own entries, one bank further each, and
// every warp picks the best candidate itself: 64 lanes x 512 keys 10.3 -> 10.0 us, x 8192 42.6 -> 40.3, against a table copied from a first one
// and a thread that went over the candidates.
template <typename C, int NW = C::NW, typename Sync = lc_block_sync>
__device__ __forceinline__ float attn_table(const float *levels, uint2 *lut, int lane, int warp, Sync sync = {}) {
    constexpr int NT = NW * 32;
    static_assert(NW <= 32, "a lane per warp's candidate");
    float gamma;
    if constexpr (!C::HILO) {
        __shared__ float cand_err[NW];
        __shared__ int cand_idx[NW];
        // gamma such that every level / gamma is (almost) exactly an f16
        const float lv0 = levels[0], lv1 = levels[1], lv2 = levels[2], lv3 = levels[3];
        const float ref = fmaxf(fmaxf(fabsf(lv0), fabsf(lv1)), fmaxf(fabsf(lv2), fabsf(lv3)));
        const float ia0 = lv0 != 0.f ? 1.0f / fabsf(lv0) : 0.f, ia1 = lv1 != 0.f ? 1.0f / fabsf(lv1) : 0.f;
        const float ia2 = lv2 != 0.f ? 1.0f / fabsf(lv2) : 0.f, ia3 = lv3 != 0.f ? 1.0f / fabsf(lv3) : 0.f;
        float best = INFINITY;
        int besti = 0;
        for (int j = threadIdx.x; j < 1024; j += NT) {
            const float gm = ref > 0.f ? ref / (1.0f + (float)j * (1.0f / 1024.0f)) : 1.0f;  // largest level -> [1, 2)
            const float inv = __frcp_rn(gm);
            float e = fabsf(__half2float(__float2half_rn(lv0 * inv)) * gm - lv0) * ia0;
            e = fmaxf(e, fabsf(__half2float(__float2half_rn(lv1 * inv)) * gm - lv1) * ia1);
            e = fmaxf(e, fabsf(__half2float(__float2half_rn(lv2 * inv)) * gm - lv2) * ia2);
            e = fmaxf(e, fabsf(__half2float(__float2half_rn(lv3 * inv)) * gm - lv3) * ia3);
            if (e < best) { best = e; besti = j; }
        }
        auto arg_min = [&](int width) {   // of the lanes, lowest index on ties
            for (int off = width / 2; off > 0; off >>= 1) {
                const float oe = __shfl_xor_sync(0xffffffffu, best, off);
                const int oi = __shfl_xor_sync(0xffffffffu, besti, off);
                if (oe < best || (oe == best && oi < besti)) { best = oe; besti = oi; }
            }
        };
        arg_min(32);
        if (lane == 0) { cand_err[warp] = best; cand_idx[warp] = besti; }
        sync();
        best = lane < NW ? cand_err[lane] : INFINITY;
        besti = lane < NW ? cand_idx[lane] : 0x7fffffff;
        arg_min(32);
        gamma = ref > 0.f ? ref / (1.0f + (float)besti * (1.0f / 1024.0f)) : 1.0f;
    } else {
        // the largest level becomes 1; each level is stored as two f16
        float ref = 0.f;
#pragma unroll
        for (int i = 0; i < (1 << C::BITS); i++) ref = fmaxf(ref, fabsf(levels[i]));
        gamma = ref > 0.f ? ref : 1.0f;
    }
    // a thread per entry, or as many as there are: they share its copies
    constexpr int SHARE = C::NENT < NT ? NT / C::NENT : 1, COPIES = SHARE < LUT_COPIES ? LUT_COPIES / SHARE : 1;
    for (int e = threadIdx.x / SHARE; e < C::NENT; e += NT / SHARE) {
        uint2 v;
        if constexpr (!C::HILO) {
            v.x = pack_h2(levels[e & 3] / gamma, levels[(e >> 2) & 3] / gamma);
            v.y = pack_h2(levels[(e >> 4) & 3] / gamma, levels[(e >> 6) & 3] / gamma);
        } else {
            constexpr int M = (1 << C::BITS) - 1;
            split_h2(levels[e & M] / gamma, levels[(e >> C::BITS) & M] / gamma, v.x, v.y);   // {two high parts, two low parts}
        }
        const int first = (threadIdx.x % SHARE) * COPIES;
        if (first < LUT_COPIES) {
#pragma unroll
            for (int c = 0; c < COPIES; c++) lut[e * LUT_COPIES + ((first + c + e) & (LUT_COPIES - 1))] = v;
        }
    }
    return gamma;
}

// The fields of two packed rows side by side: every second BITS-wide field of the word run, from the first on, of `a` next to the same
// of `b` (in lo), and those between (in hi); so a table field of two codes takes one of either row.
template <int WIDTH, int N>
__device__ __forceinline__ void pair_rows(const uint32_t (&a)[N], const uint32_t (&b)[N], uint32_t (&lo)[N], uint32_t (&hi)[N]) {
    static_for<N>([&](auto I) {
        constexpr int i = decltype(I)::value;
        constexpr uint32_t mask = [] {
            uint32_t m = 0;
            for (int j = 0; j < 32; j++)
                if ((32 * i + j) / WIDTH % 2 == 0) m |= 1u << j;
            return m;
        }();
        uint32_t up, down;   // (a field may cross into the next word)
        if constexpr (32 % (2 * WIDTH) == 0) {
            up = b[i] << WIDTH;
            down = a[i] >> WIDTH;
        } else {
            up = __funnelshift_l(i > 0 ? b[i > 0 ? i - 1 : 0] : 0u, b[i], WIDTH);
            down = __funnelshift_r(a[i], i + 1 < N ? a[i + 1 < N ? i + 1 : i] : 0u, WIDTH);
        }
        lo[i] = (a[i] & mask) | (up & ~mask);
        hi[i] = (down & mask) | (b[i] & ~mask);
    });
}

// A warp's state over its tiles: O^T fragments, running maxima of heads 2t, 2t + 1 and this thread's part of the sums.
template <typename C>
struct AttnAcc {
    float o[C::NO][4], m_run[2], l_part[2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int s = 0; s < C::NO; s++) o[s][0] = o[s][1] = o[s][2] = o[s][3] = 0.f;
        m_run[0] = m_run[1] = -INFINITY;
        l_part[0] = l_part[1] = 0.f;
    }
    // O^T of dims (HD / 8) g + 2 s (heads 2t, 2t + 1), + 1 (the same)
    __device__ __forceinline__ float4 result(int s) const {
        if constexpr (!C::PAIRS) return make_float4(o[s][0], o[s][1], o[s][2], o[s][3]);
        else if constexpr (C::HILO) return make_float4(o[2 * s][0] + o[2 * s][2], o[2 * s][1] + o[2 * s][3], o[2 * s + 1][0] + o[2 * s + 1][2], o[2 * s + 1][1] + o[2 * s + 1][3]);
        else return s % 2 == 0 ? make_float4(o[s][0], o[s][1], o[s | 1][0], o[s | 1][1]) : make_float4(o[s & ~1][2], o[s & ~1][3], o[s][2], o[s][3]);
    }
};
// One warp's step over the KT keys t0 .. t0 + KT - 1 (those below k_end count) whose codes lie at the shared-memory addresses ka
// and va.  nk, nv: norms times gamma of key `lane`.  q_a: this lane's query fragments where they stay in shared memory.
//
// A lookup's eight bytes land in two neighbouring registers, and an MMA's A operand is four in a row, of which the first two (and the last
// two) are operand rows g and g + 8 at the same k.  So what a lookup returns is arranged to be such a pair, which saves the moves and
// permutes that put operands together (15 of 54 instructions per key at 4 bits):
//   * S^T, two parts: rows g and g + 8 are the high and the low part of one key.  One part: two keys, their codes side by side (pair_rows);
//   * O^T, two parts: the high and low part of one dim, at two adjacent keys, whose codes lie side by side; the two parts' sums stay apart
//     until the end.  One part: two dims, at two adjacent keys.
// 64 lanes x 8192 keys: tq2 47.1 -> 42.6 us, tq3 95.3 -> 85.5, tq4 85.3 -> 80.0.
template <typename C, int NQ>
__device__ __forceinline__ void attn_tile(AttnAcc<C> &st, uint32_t ka, uint32_t va, uint32_t t0, uint32_t k_end, float nk, float nv,
                                          const uint32_t (&bq)[NQ][2], const uint32_t (&bql)[NQ][2], uint32_t q_a, uint32_t lut_lane, int lane) {
    constexpr int CB = C::CB, KT = C::KT, MT = C::MT, NS = C::NS, FB = C::FB, NO = C::NO;
    const int g = lane >> 2, t = lane & 3;
    float(&o)[NO][4] = st.o;
    float(&m_run)[2] = st.m_run, (&l_part)[2] = st.l_part;
    // ---- S^T[KT keys x 8 heads] ----
    constexpr int KG = KT / 8, KW = CB / 16;   // words of one key in this thread's quarter row
    float sc[KG][2];   // logits of keys 8 kg + g for heads 2t, 2t + 1, less the key's norm
    {
        uint32_t kw[KG][KW];
#pragma unroll
        for (int kg = 0; kg < KG; kg++) lds_words<KW>(ka + (uint32_t)(8 * kg + g) * C::KRS + (uint32_t)t * (KW * 4), kw[kg]);
        constexpr int NC = C::HILO ? KG : MT;
        float c[NC][2][4];   // chains: high and low query parts
#pragma unroll
        for (int i = 0; i < NC; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) c[i][0][e] = c[i][1][e] = 0.f;
        if constexpr (!C::HILO) {
            // bytes of two codes of key g and the same two of key g + 8: four dims of a k-step are a byte of either run
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                uint32_t lo[KW], hi[KW];
                pair_rows<4>(kw[2 * mt], kw[2 * mt + 1], lo, hi);
#pragma unroll
                for (int w = 0; w < KW; w++) { kw[2 * mt][w] = lo[w]; kw[2 * mt + 1][w] = hi[w]; }
            }
        }
        static_for<NS>([&](auto S) {
            constexpr int s = decltype(S)::value;
            uint32_t b0, b1, l0, l1;
            if constexpr (C::QSMEM) {
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(b0), "=r"(b1), "=r"(l0), "=r"(l1) : "r"(q_a + s * 512));
            } else {
                b0 = bq[s][0]; b1 = bq[s][1]; l0 = bql[s][0]; l1 = bql[s][1];
            }
#pragma unroll
            for (int i = 0; i < NC; i++) {
                uint2 x, y;
                if constexpr (!C::HILO) {
                    x = lds64(field_addr<FB, s * FB>(kw[2 * i], lut_lane));
                    y = lds64(field_addr<FB, s * FB>(kw[2 * i + 1], lut_lane));
                } else {
                    x = lds64(field_addr<FB, 2 * s * FB>(kw[i], lut_lane));
                    y = lds64(field_addr<FB, (2 * s + 1) * FB>(kw[i], lut_lane));
                }
                const uint32_t a[4] = {x.x, x.y, y.x, y.y};
                mma16816(c[i][0], a, b0, b1);
                mma16816(c[i][1], a, l0, l1);
            }
        });
#pragma unroll
        for (int kg = 0; kg < KG; kg++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                sc[kg][h] = C::HILO ? c[kg % NC][0][h] + (c[kg % NC][0][2 + h] + c[kg % NC][1][h] + c[kg % NC][1][2 + h])
                                    : c[kg / 2][0][2 * (kg % 2) + h] + c[kg / 2][1][2 * (kg % 2) + h];
    }

    // ---- online softmax ----
    float tm[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int kg = 0; kg < KG; kg++) {
        const int key = 8 * kg + g;
        const float kn = __shfl_sync(0xffffffffu, nk, key);
        const bool valid = t0 + key < k_end;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            sc[kg][h] = valid ? sc[kg][h] * kn : -INFINITY;
            tm[h] = fmaxf(tm[h], sc[kg][h]);
        }
    }
    float resc[2];
    // Where P has two parts the running maximum may lag by 8, so the accumulators are hardly ever rescaled: weights reach e^8, and norms
    // above 21, which could take P past an f16, move it at once.
    const float lag = C::HILO && !__any_sync(0xffffffffu, fabsf(nv) > 21.0f) ? 8.0f : 0.0f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        tm[h] = fmaxf(tm[h], __shfl_xor_sync(0xffffffffu, tm[h], 4));
        tm[h] = fmaxf(tm[h], __shfl_xor_sync(0xffffffffu, tm[h], 8));
        tm[h] = fmaxf(tm[h], __shfl_xor_sync(0xffffffffu, tm[h], 16));
        const float m_new = C::HILO ? (tm[h] > m_run[h] + lag ? tm[h] : m_run[h]) : fmaxf(m_run[h], tm[h]);    // finite: key t0 is valid
        resc[h] = soft_exp<C::HILO>(m_run[h] - m_new);
        m_run[h] = m_new;
        l_part[h] *= resc[h];
    }
    // P (times the value norms) into the B operand: (key g | g+8; heads 2t, 2t+1) -> (keys 2t, 2t+1 | +8; head g)
    uint32_t bp[MT][2], bpl[MT][2];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float vn = __shfl_sync(0xffffffffu, nv, (KT == 32 ? 16 * mt : 0) + 8 * r + g);
            const float p0 = soft_exp<C::HILO>(sc[2 * mt + r][0] - m_run[0]), p1 = soft_exp<C::HILO>(sc[2 * mt + r][1] - m_run[1]);
            l_part[0] += p0;
            l_part[1] += p1;
            if constexpr (!C::HILO) {
                bp[mt][r] = movmatrix_trans(pack_h2(p0 * vn, p1 * vn));
            } else {
                uint32_t hi, lo;
                split_h2(p0 * vn, p1 * vn, hi, lo);
                bp[mt][r] = movmatrix_trans(hi);
                bpl[mt][r] = movmatrix_trans(lo);
            }
        }
    }
    if (__any_sync(0xffffffffu, resc[0] != 1.0f || resc[1] != 1.0f)) {   // the running max moved for some head
#pragma unroll
        for (int s = 0; s < NO; s++) {
            o[s][0] *= resc[0]; o[s][1] *= resc[1]; o[s][2] *= resc[0]; o[s][3] *= resc[1];
        }
    }

    // ---- O^T[HD dims x 8 heads] += V^T . P (AttnAcc::result says which dims a tile's rows g, g + 8 are) ----
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        constexpr int VW = CB % 32 == 0 ? CB / 32 : 2;   // words of one key in this thread's eighth row
        uint32_t vw[4][VW];   // keys 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t row = va + (uint32_t)(16 * mt + 2 * t + (q & 1) + 8 * (q >> 1)) * C::VRS;
            if constexpr (CB % 32 == 0) {
                lds_words<VW>(row + (uint32_t)g * (VW * 4), vw[q]);
            } else {   // 6-byte pieces (tq3 at head_dim 128): two aligned words, shifted into place
                const uint32_t a = row + (uint32_t)g * 6u, sh = (a & 2u) * 8u;
                uint32_t w[2];
                asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w[0]) : "r"(a & ~3u));
                asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w[1]) : "r"((a & ~3u) + 4u));
                vw[q][0] = __funnelshift_r(w[0], w[1], sh);
                vw[q][1] = w[1] >> sh;
            }
        }
        if constexpr (C::PAIRS) {
            uint32_t pw[2][2][VW];   // [keys 2t .. | 2t + 8 ..][codes 0, 2, 4 .. | 1, 3, 5 ..]
#pragma unroll
            for (int q = 0; q < 2; q++) pair_rows<C::BITS>(vw[2 * q], vw[2 * q + 1], pw[q][0], pw[q][1]);
            static_for<(C::HILO ? NS : NS / 2)>([&](auto U) {   // one dim (two parts) or dims d, d + 2 of either run of codes
                constexpr int u = decltype(U)::value;
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint2 x = lds64(field_addr<FB, u * FB>(pw[0][e], lut_lane)), y = lds64(field_addr<FB, u * FB>(pw[1][e], lut_lane));
                    const uint32_t a[4] = {x.x, x.y, y.x, y.y};
                    mma16816(o[2 * u + e], a, bp[mt][0], bp[mt][1]);
                    if constexpr (C::HILO) mma16816(o[2 * u + e], a, bpl[mt][0], bpl[mt][1]);
                }
            });
        } else {
            static_for<NS>([&](auto U) {
                constexpr int u = decltype(U)::value;
                const uint2 e0 = lds64(field_addr<FB, u * FB>(vw[0], lut_lane)), e1 = lds64(field_addr<FB, u * FB>(vw[1], lut_lane));   // keys 2t, 2t+1
                const uint2 e2 = lds64(field_addr<FB, u * FB>(vw[2], lut_lane)), e3 = lds64(field_addr<FB, u * FB>(vw[3], lut_lane));   // keys 2t+8, 2t+9
                // .x: high parts of two dims; .y: low parts
                const uint32_t ax[4] = {__byte_perm(e0.x, e1.x, 0x5410), __byte_perm(e0.x, e1.x, 0x7632), __byte_perm(e2.x, e3.x, 0x5410),
                                        __byte_perm(e2.x, e3.x, 0x7632)};
                const uint32_t ay[4] = {__byte_perm(e0.y, e1.y, 0x5410), __byte_perm(e0.y, e1.y, 0x7632), __byte_perm(e2.y, e3.y, 0x5410),
                                        __byte_perm(e2.y, e3.y, 0x7632)};
                mma16816(o[u], ax, bp[mt][0], bp[mt][1]);
                mma16816(o[u], ax, bpl[mt][0], bpl[mt][1]);
                mma16816(o[u], ay, bp[mt][0], bp[mt][1]);
            });
        }
    }
}

}  // namespace
