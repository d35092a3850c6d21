// Prefill / multi-row attention over TurboQuant codes on tcgen05: head_dim 128 / 256, tq2 / tq3 / tq4.  Stands in for
// shaders/attention_flash_tq.metal:290-556 (flash_attention_tq_prefill and its query-tiled form) for chunks of several rows;
// leaves the split-K partials that a merge launch (attention_tq.cu) adds up.
//
// The decode kernel serves one query row per CTA, so a chunk of 256 rows decoded the same cache 256 times.  Here a CTA owns 128
// query rows of the MMA's M (16 tokens x 8 heads of a kv-head) and a range of keys:
//   * twelve warps (eight for K, four for V) decode KN keys at a time into f16 operand tiles in shared memory (128-byte swizzle): K and V have the same
//     layout, K is read K-major (dims contiguous), V as a transposed operand (the MMA's K runs over keys);
//   * S[128 x KN] = Q . K^T with the query as an f16 and the f16 of its remainder (two MMAs per slice), f32 in tensor memory,
//     two buffers, so the next tile's product runs beside this one's softmax;
//   * eight warps own half a query row per thread: row norms, causal and window mask, online softmax with the running maximum moved
//     only when it has grown by more than LAZY (a rescale is a pass over the accumulator), or at all where a tile's value norms
//     are so large that P could leave f16's range; P times the value norms goes back to tensor memory;
//   * O[128 x HD] += P . V with P read from tensor memory.
// Precision as in attention_tq_mma.cu: levels and P are an f16 and the f16 of the remainder, which doubles the operand tiles, but for tq2
// at head_dim 256, whose levels are f16-exact up to a factor gamma that is folded into the norms and whose P is an f16.
// Every barrier wait is bounded; on expiry the CTA records a status word and leaves.
#include <math.h>
#include <utility>

#include "attention_tq.h"
#include "tcgen05_util.cuh"

namespace {

constexpr int M = 128;
constexpr int SMW = 8, DKW = 8, DVW = 4, MMA_WARP = SMW + DKW + DVW, PF_NT = (MMA_WARP + 1) * 32;   // softmax, K, V, issue
// A weight is at most e^LAZY while the running maximum lags, and P, the weight times v_norm * gamma, is stored as f16: tiles with
// a larger factor than LAZY_VMAX (e^8 * 21 = 62600 < 65504) move the maximum whenever it grows, which leaves P <= v_norm * gamma.
// Unit normal V rows have 1 - 3, so the usual tile keeps the lag.
constexpr float LAZY = 8.0f, LAZY_VMAX = 21.0f;

template <int HD_, int BITS_>
struct PfCfg {
    static constexpr int HD = HD_, BITS = BITS_, CB = HD * BITS / 8;
    static constexpr int KN = HD == 256 && BITS > 2 ? 32 : 64;   // keys per tile (what fits beside the query)
    static constexpr int PARTS = BITS > 2 || HD != 256 ? 2 : 1;  // operand tiles per level, and parts of P: f16, remainder
    static constexpr int NB = HD / 64;                           // 64-dim blocks (128 bytes: the swizzle's width)
    static constexpr int UN = HD / 32, UB = 4 * BITS;            // 32-dim units of a row, bytes of a unit
    static constexpr int NUK = KN * UN / (DKW * 32), NUV = KN * UN / (DVW * 32);   // units per decoding thread
    static constexpr int FB = 2 * BITS, NENT = 1 << FB, COPIES = 8;   // table of two codes
    static constexpr int Q_PART = NB * M * 128, KV_PART = NB * KN * 128;
    // The query's f16 parts are A operands in tensor memory, but for the remainder at head_dim 256, which has no room there.
    // K and V tiles have two buffers each.
    static constexpr bool QL_SMEM = HD == 256;
    static constexpr int SIDE = PARTS * KV_PART;                 // one tile of K or V
    static constexpr int QL_OFF = 0, K_OFF = QL_SMEM ? Q_PART : 0, V_OFF = K_OFF + 2 * SIDE, LUT_OFF = V_OFF + 2 * SIDE;
    // Before the first tile: signed query rows (until the transform has read them), and query parts on their way to tensor memory.
    static constexpr int RAW_OFF = QL_SMEM ? QL_OFF : V_OFF, QST_OFF = K_OFF;
    static constexpr int LUT_BYTES = PARTS == 2 ? NENT * COPIES * 8 : 0;
    static constexpr int NORM_OFF = LUT_OFF + LUT_BYTES, NORM_BYTES = 4 * 2 * KN * 4;   // [4 tiles][k, v][KN]
    static constexpr int STAGE = M * (HD + 4) * 4;               // results, reuses the operand tiles
    static constexpr int TAIL = NORM_OFF + NORM_BYTES;
    static constexpr int SMEM = (TAIL > STAGE ? TAIL : STAGE) + 256 + 1024;
    static constexpr int NVW = KN / 32;                          // warps that fetch a tile's V norms, one lane per key
    static_assert(NUK >= 1 && NUV >= 1 && SMEM <= 226 * 1024, "shared memory");
    static_assert((QL_SMEM ? 1 : 2) * Q_PART <= 4 * SIDE && Q_PART <= 2 * SIDE && 64 * 128 <= 2 * SIDE, "what K's and V's place holds at first");
    // Tensor memory: S x 2 (P and its remainder replace the S they come from), the query's two parts, O.
    static constexpr int S_COL = 0, QH_COL = 128, QL_COL = 192, O_COL = 256;
    static_assert(2 * KN <= QH_COL && QH_COL + HD / 2 <= (QL_SMEM ? O_COL : QL_COL) && O_COL + HD <= 512, "tensor memory");
};

__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Operand descriptor of a tile whose rows (64 elements, 128-byte swizzle) run along the MMA's K: 1024 bytes between groups of
// eight rows, `block` bytes between blocks of 64 elements of the other dimension.
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t saddr, uint32_t block) {
    return make_desc(saddr) | (uint64_t)((block >> 4) & 0x3FFFu) << 16;
}
__device__ __forceinline__ uint32_t pack2(float x, float y) {
    const __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void split2(float x, float y, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = pack2(x - f.x, y - f.y);
}
template <int PARTS>
__device__ __forceinline__ float pf_exp(float x) { return PARTS == 1 ? __expf(x) : expf(x); }
__device__ __forceinline__ void sts16(uint32_t a, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void lds128(uint32_t a, uint32_t (&v)[4]) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
// four columns of this thread's row
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
// Walsh-Hadamard butterflies over 32 * DPL values, DPL consecutive ones per lane, ascending stride.
template <int DPL>
__device__ __forceinline__ void fwht_lanes(float (&x)[DPL], int lane) {
#pragma unroll
    for (int len = 1; len < DPL; len <<= 1)
#pragma unroll
        for (int i = 0; i < DPL; i++)
            if (!(i & len)) {
                const float a = x[i], b = x[i + len];
                x[i] = a + b;
                x[i + len] = a - b;
            }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const bool upper = lane & m;
#pragma unroll
        for (int i = 0; i < DPL; i++) {
            const float o = __shfl_xor_sync(0xffffffffu, x[i], m);
            x[i] = upper ? o - x[i] : x[i] + o;
        }
    }
}
// Where dim d of a row sits in the operand tiles: levels in one part keep the order in which a byte table decodes sixteen dims.
template <int PARTS>
__device__ __forceinline__ int tile_pos(int d) {
    return PARTS == 1 ? (d & ~15) + 4 * (d & 3) + ((d >> 2) & 3) : d;
}

template <typename C>
__global__ void __launch_bounds__(PF_NT, 1) tq_attn_prefill_kernel(const TqAttnParams p) {
    constexpr int HD = C::HD, BITS = C::BITS, KN = C::KN, NB = C::NB, DPL = HD / 32;
    lc_pdl_trigger();
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t base = smem_u32(smem);
    float *norms = reinterpret_cast<float *>(smem + C::NORM_OFF);
    constexpr int BAR_OFF = C::TAIL > C::STAGE ? C::TAIL : C::STAGE;
    const uint32_t bars = base + BAR_OFF;
    // two of each, of even and odd tiles: a side may be a tile ahead of a role that waits for it
    const uint32_t k_full = bars, v_full = bars + 16, p_full = bars + 32, pv_done = bars + 48, qk_done = bars + 64, rot_done = bars + 80;
    auto of_tile = [](uint32_t bar, int t) -> uint32_t { return bar + 8u * (uint32_t)(t & 1); };
    auto phase_of = [](int t) -> uint32_t { return (uint32_t)((t >> 1) & 1); };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + BAR_OFF + 96);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    __shared__ float m_s[M], l_s[2][M], mx_s[2][2][M], vmax_s[4][C::NVW], cand_err[PF_NT / 32];
    __shared__ int cand_idx[PF_NT / 32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t gchunks = (p.group + 7) / 8;
    const uint32_t kv_head = blockIdx.y / gchunks, gchunk = blockIdx.y - kv_head * gchunks;
    const int gvalid = min(8, (int)(p.group - gchunk * 8)), gc = (int)p.pf_heads;   // rows per token: gvalid rounded up to a power of two
    const uint32_t qh0 = kv_head * p.group + gchunk * 8;
    const int toks = M / gc, tok0 = (int)blockIdx.z * toks, nt = min(toks, (int)p.n_lanes - tok0);   // tokens of this tile
    const uint32_t split = blockIdx.x;
    // keys that any row of the tile sees, this split's share of them
    const uint32_t pos0 = p.current_pos + tok0, pos1 = pos0 + nt - 1;
    const uint32_t key_end = min(p.kv_len, pos1 + 1u);
    const uint32_t key_lo = (p.window > 0u && pos0 + 1u > p.window) ? pos0 + 1u - p.window : 0u;
    const uint32_t n_keys = key_end > key_lo ? key_end - key_lo : 0u;
    uint32_t per = (n_keys + p.n_splits - 1) / p.n_splits;
    per = (per + KN - 1) / KN * KN;
    const uint32_t k_begin = min(key_end, key_lo + split * per), k_end = min(key_end, k_begin + per);
    const int tiles = (int)((k_end - k_begin + KN - 1) / KN);

    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < 16; i += 8) {
            mbar_init(k_full + i, DKW + p.extra_arrivals);
            mbar_init(v_full + i, DVW);
            mbar_init(p_full + i, SMW);
            mbar_init(pv_done + i, 1);
            mbar_init(qk_done + i, 1);
        }
        mbar_init(rot_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // ---- levels (constant operands) ----
    float lvl[1 << BITS], ref = 0.f;
#pragma unroll
    for (int i = 0; i < (1 << BITS); i++) {
        lvl[i] = p.levels[i];
        ref = fmaxf(ref, fabsf(lvl[i]));
    }
    float gamma;
    if constexpr (C::PARTS == 1) {   // gamma such that every level / gamma is (almost) exactly an f16
        float best = INFINITY;
        int besti = 0;
        for (int j = tid; j < 1024; j += PF_NT) {
            const float gm = ref > 0.f ? ref / (1.0f + (float)j * (1.0f / 1024.0f)) : 1.0f;
            const float inv = __frcp_rn(gm);
            float e = 0.f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float ia = lvl[i] != 0.f ? 1.0f / fabsf(lvl[i]) : 0.f;
                e = fmaxf(e, fabsf(__half2float(__float2half_rn(lvl[i] * inv)) * gm - lvl[i]) * ia);
            }
            if (e < best) { best = e; besti = j; }
        }
        auto arg_min = [&]() {   // of the lanes, lowest index on ties
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const float oe = __shfl_xor_sync(0xffffffffu, best, off);
                const int oi = __shfl_xor_sync(0xffffffffu, besti, off);
                if (oe < best || (oe == best && oi < besti)) { best = oe; besti = oi; }
            }
        };
        arg_min();
        if (lane == 0) { cand_err[warp] = best; cand_idx[warp] = besti; }
        __syncthreads();
        static_assert(PF_NT / 32 <= 32, "a lane per warp's candidate");
        best = lane < PF_NT / 32 ? cand_err[lane] : INFINITY;   // every warp by itself (256 rows over 4096 keys 29.5 -> 29.3 us against a thread that goes over them)
        besti = lane < PF_NT / 32 ? cand_idx[lane] : 0x7fffffff;
        arg_min();
        gamma = ref > 0.f ? ref / (1.0f + (float)besti * (1.0f / 1024.0f)) : 1.0f;
    } else {
        gamma = ref > 0.f ? ref : 1.0f;
        uint2 *lut = reinterpret_cast<uint2 *>(smem + C::LUT_OFF);
        for (int e = tid; e < C::NENT * C::COPIES; e += PF_NT) {
            const int c = e / C::COPIES;
            uint2 v;
            split2(p.levels[c & ((1 << BITS) - 1)] / gamma, p.levels[(c >> BITS) & ((1 << BITS) - 1)] / gamma, v.x, v.y);
            lut[e] = v;
        }
    }
    lc_pdl_wait();

    // ---- query rows: sign, transform, scale, split into two f16 operand tiles (K-major, 128-byte swizzle) ----
    auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool { return mbar_wait_warp(bar, parity, p.wait_limit, abort_flag); };
    // The transform of 128 rows by shuffles took 13 of this kernel's 61 thousand cycles (16 rows over 2000 keys 21.0 -> 19.1 us
    // without it, 256 over 4096 39.4 -> 37.8).  With signs of +-1 the signed row is an f16 still, exactly, and 64 dims of it at a
    // time go through the tensor cores: D = A . H64 (Sylvester's matrix, its rows in the order of the operand tiles), then butterflies over the 64-dim blocks when a row is read back.
    bool unit = p.fused_q != 0u;
    uint32_t flip[DPL / 2];
    if (p.fused_q) {
#pragma unroll
        for (int i = 0; i < DPL; i += 2) {
            const float2 sg = *reinterpret_cast<const float2 *>(p.signs + DPL * lane + i);
            unit = unit && fabsf(sg.x) == 1.0f && fabsf(sg.y) == 1.0f;
            flip[i / 2] = (sg.x < 0.f ? 0x8000u : 0u) | (sg.y < 0.f ? 0x80000000u : 0u);
        }
    }
    unit = __all_sync(0xffffffffu, unit);   // (every warp sees all signs)
    if (unit) {
        if (warp < MMA_WARP) {
            constexpr int QB = 4;   // rows of a warp whose loads are in flight together
#pragma unroll 1
            for (int rb = warp; rb < M; rb += MMA_WARP * QB) {
                uint2 raw[QB][DPL / 4];
#pragma unroll
                for (int j = 0; j < QB; j++) {
                    const int r = rb + j * MMA_WARP, tk = r / gc, h = r - tk * gc;
#pragma unroll
                    for (int i = 0; i < DPL / 4; i++) {
                        raw[j][i] = make_uint2(0u, 0u);
                        if (r < M && tk < nt && h < gvalid)
                            raw[j][i] = *reinterpret_cast<const uint2 *>(p.q + ((size_t)(tok0 + tk) * p.n_q + qh0 + h) * HD + DPL * lane + 4 * i);
                    }
                }
#pragma unroll
                for (int j = 0; j < QB; j++) {
                    const int r = rb + j * MMA_WARP;
                    if (r >= M) break;
#pragma unroll
                    for (int i = 0; i < DPL / 4; i++) {
                        const int d = DPL * lane + 4 * i;
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(base + (uint32_t)(C::RAW_OFF + (d >> 6) * M * 128 + r * 128 + ((((d & 63) >> 3) ^ (r & 7)) << 4) + (d & 4) * 2)),
                                     "r"(raw[j][i].x ^ flip[2 * i]), "r"(raw[j][i].y ^ flip[2 * i + 1])
                                     : "memory");
                    }
                }
            }
        }
        for (int e = tid; e < 64 * 8; e += PF_NT) {   // H64 in the place of the first keys: row n is output dim tile_pos(n) (its own inverse)
            const int n = e >> 3, c = e & 7, d = tile_pos<C::PARTS>(n);
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int k = 8 * c + 2 * i;
                v[i] = ((__popc(d & k) & 1) ? 0xBC00u : 0x3C00u) | ((__popc(d & (k + 1)) & 1) ? 0xBC000000u : 0x3C000000u);
            }
            sts16(base + (uint32_t)(C::K_OFF + n * 128 + ((c ^ (n & 7)) << 4)), v);
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t d_tmem = *tmem_slot + (uint32_t)C::O_COL;
        if (warp == MMA_WARP) {
            const bool leader = elect_one();
            const uint32_t idesc = (1u << 4) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
            if (leader) {
#pragma unroll
                for (int nb = 0; nb < NB; nb++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        umma_ss(d_tmem + 64u * nb, make_desc(base + C::RAW_OFF + nb * M * 128) + 2 * j, make_desc(base + C::K_OFF) + 2 * j, idesc, j > 0 ? 1u : 0u);
                umma_commit(rot_done);
            }
            __syncwarp();
        }
        if (warp < SMW) {   // two threads per row, half of each block's columns each
            const int half = warp >> 2, r = (warp & 3) * 32 + lane;
            const uint32_t tq = d_tmem + ((uint32_t)(32 * (warp & 3)) << 16);
            const float f = p.scale / sqrtf((float)HD);
            warp_wait(rot_done, 0u);
            tc_fence_after();
#pragma unroll 1
            for (int c = 4 * half; c < 4 * half + 4; c++) {
                uint32_t v[NB][8];
#pragma unroll
                for (int nb = 0; nb < NB; nb++) tmem_ld8(tq + (uint32_t)(64 * nb + 8 * c), v[nb]);
                tmem_ld_wait();
#pragma unroll
                for (int len = 1; len < NB; len <<= 1)
#pragma unroll
                    for (int nb = 0; nb < NB; nb++)
                        if (!(nb & len)) {
#pragma unroll
                            for (int i = 0; i < 8; i++) {
                                const float a = __uint_as_float(v[nb][i]), b = __uint_as_float(v[nb + len][i]);
                                v[nb][i] = __float_as_uint(a + b);
                                v[nb + len][i] = __float_as_uint(a - b);
                            }
                        }
#pragma unroll
                for (int nb = 0; nb < NB; nb++) {
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) split2(__uint_as_float(v[nb][2 * i]) * f, __uint_as_float(v[nb][2 * i + 1]) * f, hi[i], lo[i]);
                    tmem_st4(tq - C::O_COL + C::QH_COL + 32 * nb + 4 * c, hi);
                    if (C::QL_SMEM) sts16(base + (uint32_t)(C::QL_OFF + nb * M * 128 + r * 128 + ((c ^ (r & 7)) << 4)), lo);
                    else tmem_st4(tq - C::O_COL + C::QL_COL + 32 * nb + 4 * c, lo);
                }
            }
            tmem_st_wait();
        }
    } else if (warp < MMA_WARP) {   // queries rotated already, or other signs
#pragma unroll 1
        for (int r = warp; r < M; r += MMA_WARP) {
            const int tk = r / gc, h = r - tk * gc;
            float x[DPL];
#pragma unroll
            for (int i = 0; i < DPL; i++) x[i] = 0.f;
            if (tk < nt && h < gvalid) {
                if (p.fused_q) {
#pragma unroll
                    for (int i = 0; i < DPL; i += 4) {
                        const uint2 q4 = *reinterpret_cast<const uint2 *>(p.q + ((size_t)(tok0 + tk) * p.n_q + qh0 + h) * HD + DPL * lane + i);
                        const float4 sg = *reinterpret_cast<const float4 *>(p.signs + DPL * lane + i);
                        const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&q4.x)), f1 = __half22float2(*reinterpret_cast<const __half2 *>(&q4.y));
                        x[i] = f0.x * sg.x;
                        x[i + 1] = f0.y * sg.y;
                        x[i + 2] = f1.x * sg.z;
                        x[i + 3] = f1.y * sg.w;
                    }
                    fwht_lanes<DPL>(x, lane);
                    const float f = p.scale / sqrtf((float)HD);
#pragma unroll
                    for (int i = 0; i < DPL; i++) x[i] *= f;
                } else {
                    const size_t q_row = ((size_t)(tok0 + tk) * p.n_q + qh0 + h) * HD + DPL * lane;
#pragma unroll
                    for (int i = 0; i < DPL; i += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(p.rq + q_row + i);
                        x[i] = v.x * p.scale;
                        x[i + 1] = v.y * p.scale;
                        x[i + 2] = v.z * p.scale;
                        x[i + 3] = v.w * p.scale;
                    }
                }
            }
            // levels in one part: sixteen dims (two lanes') are stored in the order 4 (d % 4) + d / 4
            if constexpr (C::PARTS == 1 && DPL == 8) {   // the even lane takes dims d % 4 = 0, 1 of both, the odd lane 2, 3
                const bool odd = lane & 1;
                float y[8];
#pragma unroll
                for (int l = 0; l < 2; l++)
#pragma unroll
                    for (int bb = 0; bb < 2; bb++) {
                        const float mine = odd ? x[4 * bb + 2 + l] : x[4 * bb + l], give = odd ? x[4 * bb + l] : x[4 * bb + 2 + l];
                        const float got = __shfl_xor_sync(0xffffffffu, give, 1);
                        y[4 * l + bb] = odd ? got : mine;
                        y[4 * l + 2 + bb] = odd ? mine : got;
                    }
#pragma unroll
                for (int i = 0; i < 8; i++) x[i] = y[i];
            }
            if constexpr (DPL == 8) {   // a lane's eight values are one 16-byte chunk
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int i = 0; i < 4; i++) split2(x[2 * i], x[2 * i + 1], hi[i], lo[i]);
                const uint32_t off = base + (uint32_t)((lane >> 3) * M * 128 + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                sts16(off + C::QST_OFF, hi);
                sts16(off + (C::QL_SMEM ? C::QL_OFF : C::QST_OFF + C::Q_PART), lo);
            } else {
#pragma unroll
                for (int i = 0; i < DPL; i++) {
                    const int pos = tile_pos<C::PARTS>(DPL * lane + i), nb = pos >> 6, c = (pos & 63) >> 3;
                    const uint32_t off = (uint32_t)(nb * M * 128 + r * 128 + ((c ^ (r & 7)) << 4) + (pos & 7) * 2);
                    const __half hi = __float2half_rn(x[i]), lo = __float2half_rn(x[i] - __half2float(hi));
                    *reinterpret_cast<__half *>(smem + C::QST_OFF + off) = hi;
                    *reinterpret_cast<__half *>(smem + (C::QL_SMEM ? C::QL_OFF : C::QST_OFF + C::Q_PART) + off) = lo;
                }
            }
        }
    }
    if (!unit) {   // (the same for every warp)
        __syncthreads();
        if (warp < SMW) {   // into tensor memory: two threads per row, half of each block's columns each
            const int half = warp >> 2, r = (warp & 3) * 32 + lane;
            const uint32_t tq = *tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll 1
            for (int e = 0; e < 4 * NB; e++) {
                const int nb = e >> 2, c = 4 * half + (e & 3);
                const uint32_t off = base + (uint32_t)(C::QST_OFF + nb * M * 128 + r * 128 + ((c ^ (r & 7)) << 4));
                uint32_t v[4];
                lds128(off, v);
                tmem_st4(tq + C::QH_COL + 32 * nb + 4 * c, v);
                if (!C::QL_SMEM) {
                    lds128(off + C::Q_PART, v);
                    tmem_st4(tq + C::QL_COL + 32 * nb + 4 * c, v);
                }
            }
            tmem_st_wait();
        }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    float m_ref = -INFINITY, l_sum = 0.f;   // softmax threads: reference maximum and sum of this thread's row
    // =========================== decoding warps: codes -> f16 operand tiles ===========================
    // One side (K or V) by WARPS warps from warp `first`, into two buffers at `tiles_at`: `read` completes when a tile has been read,
    // `full` when one is in place.
    auto decode_side = [&](auto WARPS, int first, const uint8_t *codes, bool with_norms, uint32_t tiles_at, uint32_t full, uint32_t read) {
        constexpr int ND = decltype(WARPS)::value * 32, NU = KN * C::UN / ND, W = C::UB / 4;   // threads, units of a thread, words of a unit
        const int dt = tid - first * 32;
        uint32_t raw[NU][W];
        float norm_next = 0.f;
        auto slot_of = [&](uint32_t key) -> size_t { return (size_t)(p.ring ? key % p.ring : key) * p.n_kv + kv_head; };
        // unit u of a tile: key (u & 7) + 8 (u / (8 UN)), 32-dim unit (u / 8) % UN: eight lanes store to eight different rows
        auto fetch = [&](int t) {
            const uint32_t t0 = k_begin + (uint32_t)t * KN;
#pragma unroll
            for (int j = 0; j < NU; j++) {
                const int u = dt + j * ND, key = (u & 7) | ((u / (8 * C::UN)) << 3), unit = (u >> 3) % C::UN;
                const size_t s = slot_of(t0 + key < k_end ? t0 + key : t0) * C::CB + (size_t)(unit * C::UB);
                if constexpr (W == 2) {
                    const uint2 a = *reinterpret_cast<const uint2 *>(codes + s);
                    raw[j][0] = a.x; raw[j][1] = a.y;
                } else if constexpr (W == 4) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(codes + s);
                    raw[j][0] = a.x; raw[j][1] = a.y; raw[j][2] = a.z; raw[j][3] = a.w;
                } else {
#pragma unroll
                    for (int i = 0; i < W; i++) raw[j][i] = *reinterpret_cast<const uint32_t *>(codes + s + 4 * i);
                }
            }
            if (with_norms && dt < 2 * KN) {   // [k norms][v norms]
                const uint32_t key = t0 + (uint32_t)(dt % KN);
                norm_next = key < k_end ? __half2float((dt < KN ? p.kn : p.vn)[slot_of(key)]) * gamma : 0.f;
            }
        };
        [[maybe_unused]] uint32_t lut_lo = 0, lut_hi = 0;   // one part: the four levels as a byte table for prmt
        if constexpr (C::PARTS == 1) {
            const uint32_t l01 = pack2(lvl[0] / gamma, lvl[1] / gamma), l23 = pack2(lvl[2] / gamma, lvl[3] / gamma);
            lut_lo = __byte_perm(l01, l23, 0x6420);
            lut_hi = __byte_perm(l01, l23, 0x7531);
        }
        [[maybe_unused]] const uint32_t lut_lane = base + (uint32_t)C::LUT_OFF + (uint32_t)(lane & (C::COPIES - 1)) * 8u;
        auto decode = [&](const uint32_t (&raw)[NU][W], uint32_t tile) {
#pragma unroll
            for (int j = 0; j < NU; j++) {
                const int u = dt + j * ND, key = (u & 7) | ((u / (8 * C::UN)) << 3), unit = (u >> 3) % C::UN;
                const uint32_t row = tile + (uint32_t)((unit >> 1) * (KN * 128) + key * 128), c0 = (uint32_t)(unit & 1) * 4u, sw = (uint32_t)key & 7u;
                if constexpr (C::PARTS == 1) {
#pragma unroll
                    for (int w = 0; w < 2; w++) {
                        uint32_t v[8];   // sixteen dims: bit pair l of each byte, l = 0..3
#pragma unroll
                        for (int l = 0; l < 4; l++) {
                            const uint32_t sel = ((raw[j][w] >> (2 * l)) & 0x03030303u) * 0x11u + 0x40404040u;
                            v[2 * l] = __byte_perm(lut_lo, lut_hi, sel);
                            v[2 * l + 1] = __byte_perm(lut_lo, lut_hi, sel >> 16);
                        }
                        const uint32_t lo[4] = {v[0], v[1], v[2], v[3]}, hi[4] = {v[4], v[5], v[6], v[7]};
                        sts16(row + (((c0 + 2 * w) ^ sw) << 4), lo);
                        sts16(row + (((c0 + 2 * w + 1) ^ sw) << 4), hi);
                    }
                } else {
                    auto chunk = [&](auto CI) {   // eight dims: four table entries {high parts, low parts}
                        constexpr int ci = decltype(CI)::value;
                        uint32_t hi[4], lo[4];
                        auto field = [&](auto FI) {
                            constexpr int f = decltype(FI)::value, o = (4 * ci + f) * C::FB, i = o / 32, b = o % 32;
                            uint32_t x;
                            if constexpr (b + C::FB > 32) x = __funnelshift_r(raw[j][i], raw[j][i + 1 < W ? i + 1 : i], b);
                            else x = raw[j][i] >> b;
                            const uint2 e = lds64(lut_lane + (x & ((1u << C::FB) - 1u)) * (uint32_t)(C::COPIES * 8));
                            hi[f] = e.x;
                            lo[f] = e.y;
                        };
                        field(std::integral_constant<int, 0>{});
                        field(std::integral_constant<int, 1>{});
                        field(std::integral_constant<int, 2>{});
                        field(std::integral_constant<int, 3>{});
                        const uint32_t at = row + (((c0 + ci) ^ sw) << 4);
                        sts16(at, hi);
                        sts16(at + C::KV_PART, lo);
                    };
                    chunk(std::integral_constant<int, 0>{});
                    chunk(std::integral_constant<int, 1>{});
                    chunk(std::integral_constant<int, 2>{});
                    chunk(std::integral_constant<int, 3>{});
                }
            }
        };
        if (tiles > 0) fetch(0);
        for (int t = 0; t < tiles; t++) {
            uint32_t now[NU][W];
#pragma unroll
            for (int j = 0; j < NU; j++)
#pragma unroll
                for (int i = 0; i < W; i++) now[j][i] = raw[j][i];
            const float norm_now = norm_next;
            if (t + 1 < tiles) fetch(t + 1);
            if (t > 1 && !warp_wait(of_tile(read, t), phase_of(t - 2))) break;
            if (with_norms && dt < 2 * KN) {   // (QK of tile t - 2 was issued after P of tile t - 4 was there: nobody reads that tile's norms)
                norms[(t & 3) * 2 * KN + dt] = norm_now;
                if (dt >= KN) {   // whole warps: the largest magnitude (as integers, so that a NaN is the largest)
                    const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(norm_now)));
                    if (lane == 0) vmax_s[t & 3][(dt - KN) / 32] = __uint_as_float(most);
                }
            }
            decode(now, tiles_at + (uint32_t)((t & 1) * C::SIDE));
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(of_tile(full, t));
        }
    };
    if (warp >= SMW && warp < SMW + DKW) {
        decode_side(std::integral_constant<int, DKW>{}, SMW, p.kc, true, base + (uint32_t)C::K_OFF, k_full, qk_done);
    } else if (warp >= SMW + DKW && warp < MMA_WARP) {
        decode_side(std::integral_constant<int, DVW>{}, SMW + DKW, p.vc, false, base + (uint32_t)C::V_OFF, v_full, pv_done);
    } else if (warp == MMA_WARP) {
        // =========================== MMA issue ===========================
        // The whole warp runs the loop, so that descriptors stay in uniform registers; one lane issues (33 cycles per MMA at
        // N = 64 instead of 46 for a loop of one lane).
        const bool leader = elect_one();
        if (tiles > 0) {
            const uint32_t id_qk = (1u << 4) | ((uint32_t)(KN >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
            const uint32_t id_pv = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(M >> 4) << 24);   // B transposed
            bool dead = false;
            auto qk = [&](int t) {
                if (!warp_wait(of_tile(k_full, t), phase_of(t))) { dead = true; return; }
                // S of tile t takes the place of P of tile t - 2, which PV reads
                if (t > 1 && !warp_wait(of_tile(pv_done, t), phase_of(t - 2))) { dead = true; return; }
                tc_fence_after();
                const uint32_t s = tmem + (uint32_t)(C::S_COL + (t & 1) * KN), k_at = base + (uint32_t)(C::K_OFF + (t & 1) * C::SIDE);
#pragma unroll
                for (int nb = 0; nb < NB; nb++) {
                    const uint64_t ql = make_desc(base + C::QL_OFF + nb * M * 128), kh = make_desc(k_at + nb * KN * 128), kl = make_desc(k_at + C::KV_PART + nb * KN * 128);
#pragma unroll
                    for (int j = 0; j < 4; j++) {   // K = 16 slices: 32 bytes of the rows, eight columns of tensor memory
                        if (leader) {
                            const uint32_t qc = tmem + (uint32_t)(C::QH_COL + 32 * nb + 8 * j);
                            umma_f16_ta(s, qc, kh + 2 * j, id_qk, nb > 0 || j > 0 ? 1u : 0u);
                            if constexpr (C::QL_SMEM) umma_ss(s, ql + 2 * j, kh + 2 * j, id_qk, 1u);
                            else umma_f16_ta(s, qc - C::QH_COL + C::QL_COL, kh + 2 * j, id_qk, 1u);
                            if (C::PARTS == 2) umma_f16_ta(s, qc, kl + 2 * j, id_qk, 1u);
                        }
                    }
                }
                if (leader) umma_commit(of_tile(qk_done, t));
                __syncwarp();
            };
            qk(0);
            for (int t = 0; t < tiles && !dead; t++) {
                if (t + 1 < tiles) qk(t + 1);
                if (dead || !warp_wait(of_tile(v_full, t), phase_of(t)) || !warp_wait(of_tile(p_full, t), phase_of(t))) { dead = true; break; }
                tc_fence_after();
                const uint32_t v_at = base + (uint32_t)(C::V_OFF + (t & 1) * C::SIDE), pc = tmem + (uint32_t)(C::S_COL + (t & 1) * KN);
                const uint64_t vh = make_desc_mn(v_at, KN * 128), vl = make_desc_mn(v_at + C::KV_PART, KN * 128);
#pragma unroll
                for (int j = 0; j < KN / 16; j++) {   // K = 16 keys: two groups of eight rows
                    const uint64_t off = (uint64_t)(2048 >> 4) * j;
                    if (leader) {
                        umma_f16_ta(tmem + C::O_COL, pc + 8 * j, vh + off, id_pv, t > 0 || j > 0 ? 1u : 0u);
                        if (C::PARTS == 2) umma_f16_ta(tmem + C::O_COL, pc + KN / 2 + 8 * j, vh + off, id_pv, 1u);
                        if (C::PARTS == 2) umma_f16_ta(tmem + C::O_COL, pc + 8 * j, vl + off, id_pv, 1u);
                    }
                }
                if (leader) umma_commit(of_tile(pv_done, t));
                __syncwarp();
            }
            if (!dead) dead = !warp_wait(of_tile(pv_done, tiles - 1), phase_of(tiles - 1));
            if (dead) *abort_flag = 1;
        }
        __syncwarp();
    } else {
        // =========================== softmax: half a query row per thread ===========================
        // Warps w and w + 4 own the same 32 rows (a warp reads its own lane quarter of tensor memory) and half the columns each.
        constexpr int KH = KN / 2;
        const int half = warp >> 2, r = (warp & 3) * 32 + lane, tk = r / gc;
        const uint32_t pos = pos0 + (uint32_t)tk;
        const uint32_t row_end = tk < nt ? min(p.kv_len, pos + 1u) : 0u;
        const uint32_t row_lo = (p.window > 0u && pos + 1u > p.window) ? pos + 1u - p.window : 0u;
        const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        // (an expired wait does not leave the loop: the other softmax warps count on this one at their barrier)
        for (int t = 0; t < tiles; t++) {
            warp_wait(of_tile(qk_done, t), phase_of(t));
            tc_fence_after();
            float s[KH];
            {
                uint32_t v[KH / 16][16];
#pragma unroll
                for (int c = 0; c < KH / 16; c++) tmem_ld16(tq + (uint32_t)(C::S_COL + (t & 1) * KN + half * KH + 16 * c), v[c]);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < KH; i++) s[i] = __uint_as_float(v[i / 16][i % 16]);
            }
            const float *kn = norms + (t & 3) * 2 * KN + half * KH, *vn = kn + KN;
            const uint32_t t0 = k_begin + (uint32_t)(t * KN + half * KH), end = min(row_end, k_end);
            const bool in_range = vmax_s[t & 3][0] <= LAZY_VMAX && vmax_s[t & 3][C::NVW - 1] <= LAZY_VMAX;
            const float lag = in_range ? LAZY : 0.f;
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < KH; i += 4) {
                const float4 n4 = *reinterpret_cast<const float4 *>(kn + i);
                s[i] *= n4.x; s[i + 1] *= n4.y; s[i + 2] *= n4.z; s[i + 3] *= n4.w;
            }
            if (__any_sync(0xffffffffu, t0 < row_lo || t0 + KH > end)) {   // some row of the warp does not see all of it
#pragma unroll
                for (int i = 0; i < KH; i++)
                    if (t0 + i < row_lo || t0 + i >= end) s[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < KH; i++) mx = fmaxf(mx, s[i]);
            // the row's other half (two buffers: a warp may be a tile ahead)
            mx_s[t & 1][half][r] = mx;
            tc_fence_before();
            asm volatile("bar.sync 1, %0;\n" ::"n"(SMW * 32) : "memory");
            tc_fence_after();
            mx = fmaxf(mx, mx_s[t & 1][half ^ 1][r]);
            if (t == 0) {
                m_ref = mx;
            } else if (__any_sync(0xffffffffu, mx > m_ref + lag)) {
                // the accumulator moves to the new maximum: PV of the tile before has to be complete
                warp_wait(of_tile(pv_done, t - 1), phase_of(t - 1));
                tc_fence_after();
                const float m_new = fmaxf(m_ref, mx), f = m_ref == -INFINITY ? 0.f : pf_exp<C::PARTS>(m_ref - m_new);
#pragma unroll 1
                for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 16) {
                    uint32_t v[16];
                    tmem_ld16(tq + (uint32_t)(C::O_COL + c), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
                    tmem_st16(tq + (uint32_t)(C::O_COL + c), v);
                }
                tmem_st_wait();
                l_sum *= f;
                m_ref = m_new;
            }
            const float mu = m_ref == -INFINITY ? 0.f : m_ref;   // (a row that has seen no key yet)
            uint32_t ph[KH / 2], pl[C::PARTS == 2 ? KH / 2 : 1];
#pragma unroll
            for (int i = 0; i < KH; i += 4) {
                const float4 n4 = *reinterpret_cast<const float4 *>(vn + i);
                const float e0 = pf_exp<C::PARTS>(s[i] - mu), e1 = pf_exp<C::PARTS>(s[i + 1] - mu), e2 = pf_exp<C::PARTS>(s[i + 2] - mu), e3 = pf_exp<C::PARTS>(s[i + 3] - mu);
                l_sum += (e0 + e1) + (e2 + e3);
                if (C::PARTS == 2) {
                    split2(e0 * n4.x, e1 * n4.y, ph[i / 2], pl[i / 2]);
                    split2(e2 * n4.z, e3 * n4.w, ph[i / 2 + 1], pl[i / 2 + 1]);
                } else {
                    ph[i / 2] = pack2(e0 * n4.x, e1 * n4.y);
                    ph[i / 2 + 1] = pack2(e2 * n4.z, e3 * n4.w);
                }
            }
            // P in the place of S, which every softmax warp has read (the barrier above)
            const uint32_t pc = tq + (uint32_t)(C::S_COL + (t & 1) * KN + half * (KH / 2));
#pragma unroll
            for (int c = 0; c < KH / 2; c += 8) {
                uint32_t v[8];
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = ph[c + i];
                tmem_st8(pc + c, v);
                if constexpr (C::PARTS == 2) {
#pragma unroll
                    for (int i = 0; i < 8; i++) v[i] = pl[c + i];
                    tmem_st8(pc + KN / 2 + c, v);
                }
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(of_tile(p_full, t));
        }
        if (half == 0) m_s[r] = m_ref;
        l_s[half][r] = l_sum;
    }
    tc_fence_before();
    __syncthreads();   // the issuing warp has seen the last product complete
    tc_fence_after();
    const bool failed = *abort_flag != 0;
    // ---- this split's partials: through shared memory, so that rows leave as contiguous pieces ----
    float *stage = reinterpret_cast<float *>(smem);   // [M][HD + 4]
    if (warp < SMW) {
        const int half = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll 2
        for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 16) {
            uint32_t v[16];
            if (!failed && tiles > 0) {
                tmem_ld16(tq + (uint32_t)(C::O_COL + c), v);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = 0u;
            }
            // sixteen columns are sixteen dims; levels in one part keep them in the order 4 (i % 4) + i / 4
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; e++) o[e] = C::PARTS == 1 ? v[4 * e + q] : v[4 * q + e];
                sts16(base + (uint32_t)((r * (HD + 4) + c + 4 * q) * 4), o);
            }
        }
    }
    __syncthreads();
    if (!failed) {
        for (int r = warp; r < nt * gc; r += PF_NT / 32) {
            const int tk = r / gc, h = r - tk * gc;
            if (h >= gvalid) continue;
            float *dst = p.partial + (((size_t)(tok0 + tk) * p.n_q + qh0 + h) * p.n_splits + split) * (size_t)(HD + 2);
            if (lane == 0) *reinterpret_cast<float2 *>(dst) = make_float2(m_s[r], l_s[0][r] + l_s[1][r]);
#pragma unroll
            for (int i = 0; i < HD / 64; i++)
                *reinterpret_cast<float2 *>(dst + 2 + 64 * i + 2 * lane) = *reinterpret_cast<const float2 *>(stage + r * (HD + 4) + 64 * i + 2 * lane);
        }
    } else {
        tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, tid);
    }
    if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
}

template <typename C>
int launch_pf(lc_batch *b, const TqAttnParams &p, dim3 grid) {
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(tq_attn_prefill_kernel<C>, optin, b->ctx, C::SMEM));
    LC_LAUNCH_CHECKED(lc_launch(tq_attn_prefill_kernel<C>, grid, dim3(PF_NT), C::SMEM, b, p));
    b->dispatch_count++;
    return LC_OK;
}

}  // namespace

uint32_t lc_tq_attn_prefill_tile_keys(uint32_t hd, uint32_t bits) { return hd == 256 && bits > 2 ? 32u : 64u; }
bool lc_tq_attn_prefill_supported(uint32_t hd, uint32_t bits) { return (hd == 128 || hd == 256) && bits >= 2 && bits <= 4; }

int lc_tq_attn_prefill_launch(lc_batch *b, const TqAttnParams &p, dim3 grid, uint32_t hd, uint32_t bits) {
    if (hd == 128) {
        switch (bits) {
            case 2: return launch_pf<PfCfg<128, 2>>(b, p, grid);
            case 3: return launch_pf<PfCfg<128, 3>>(b, p, grid);
            default: return launch_pf<PfCfg<128, 4>>(b, p, grid);
        }
    }
    switch (bits) {
        case 2: return launch_pf<PfCfg<256, 2>>(b, p, grid);
        case 3: return launch_pf<PfCfg<256, 3>>(b, p, grid);
        default: return launch_pf<PfCfg<256, 4>>(b, p, grid);
    }
}
