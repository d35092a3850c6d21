// All layers of a decode step for one to four lanes in one launch (the sequence of decode_step.cu's run_layers between the
// embedding and the vocabulary projection; local-engine/src/layer.rs:731-868).
//
// At these batch sizes a layer is 9 MB of weights and a few rows of activations: 1.4 us of HBM time, but eight launches in a
// chain, about 4 us each, most of it hand-over (drain, dependency wait, instruction fetch).  Here one CTA per SM stays for the
// whole step and the launches become phases that hand their rows to each other through memory:
//   norms, Q/K/V | attention over splits of the keys, K and V rows encoded on the way | merge of the splits | O | norms, gate, up | down
//   * Every exchange buffer is written once per step, in 16-byte pieces, and starts out as all ones, which no piece of data is (f16
//     and f32 conversions give no such NaN).  A consumer reads the pieces it needs until they are there.  There is no fence and no
//     second trip for the data, and nothing is written twice, so nothing can be overwritten early.  (148 CTAs that post 32 bytes each
//     and read all of them: 1960 cycles; 3050 with a counter, a release by every producer and an acquire by every consumer, since
//     a fence waits for the stores' acknowledgements.)
//   * The weights of a phase are brought into shared memory by bulk copies while the phases before it run (two regions: one for
//     Q/K/V and gate/up, one for O and down), so HBM is read while the chain of small phases waits on itself.
//   * The residual stream lives in every CTA's shared memory: each computes the norms of all rows itself from the projection's
//     output, which takes two launches out of the chain.
//   * Queries are normalised, turned, rotated and split where attention needs them, and the newest key is a split of its
//     own, whose CTA encodes the row first: the KV-write launch is gone from the chain, too.
//   * Code is kept short, its loops rolled: what a layer runs through once comes out of the instruction caches at one instruction
//     per cycle from 8 KB, per 1.5 to 2.4 cycles from 16 to 32 KB and per 6 cycles from 64 KB (measured with straight runs of FFMA),
//     whatever the number of warps.
// What bounds it: latency, twelve times a layer (load, multiply, add up, post), about 23 us a layer.  35 layers at context 8192, with
// the vocabulary and the greedy choice, as launches and as one: 1143 and 878 us for one lane, 1147 and 883 for two, 1163 and 967 for three, 1159
// and 991 for four.  At eight lanes the launches are ahead, 1258 us against 1270 when that was measured (the norms of eight rows in every
// CTA, and the gate's rows, 98 KB, into each): the line lies at four, and for long contexts below (launches_faster).
// The arithmetic and its f16 rounding points are those of the launches; sums may be added in another order.
#include <math.h>
#include <stdlib.h>

#include "attention_tq_wide.cuh"
#include "qm_codes.cuh"
#include "step_small.h"
#include "tq_rows.cuh"

namespace {

constexpr int ST_NW = 16, ST_NT = ST_NW * 32, UNIT = 128, HD = 256;   // working warps; one more fetches
constexpr int PROW = 260;              // floats of a head's partial: {max, sum, -, -}, 256 sums
constexpr int MAX_HIDDEN = 2048;       // two 16-byte pieces of a row per thread at four lanes
constexpr int RED_COL = 20, RED_PART = 8 * RED_COL + 16;   // a warp's sums of a tile, floats: [column][16 rows + padding] + padding
constexpr int MAX_TILES = 16;          // of a CTA in one phase
constexpr int FEW_SPLITS = 32, FULL_SPLIT = 4;   // more splits than the former only with this many blocks of keys in each

// The exchange buffers of a layer: the counts of posts to O and to down (128 bytes each), rows of Q, K, V; attention; O; down;
// gate * up; partials.
constexpr int Q_M = 0, K_M = 1, V_M = 2, ATTN_M = 3, O_M = 4, DOWN_M = 5, GATE_M = 6, PART_M = 7, COUNTS = 256;
__host__ __device__ __forceinline__ size_t mail_rows_bytes(int m, int H, int I, int n_q, int n_kv) {
    return COUNTS + (size_t)m * 2 * ((size_t)(2 * n_q + 2 * n_kv) * HD + 2 * (size_t)H + I);
}
__host__ __device__ __forceinline__ size_t mail_partial_bytes(int m, int n_q, int splits) { return (size_t)m * n_q * (splits + 1) * PROW * 4; }

__host__ __device__ constexpr int stages_of(int bits) { return bits == 2 ? 5 : 3; }   // blocks of 64 keys in shared memory; a block less in flight

__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
// 16 bytes at once, past the first-level cache
__device__ __forceinline__ uint4 take16(const void *p) {
    uint64_t lo, hi;
    asm volatile("{\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%2];\n\tmov.b128 {%0, %1}, v;\n\t}\n" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ void post16(void *p, const uint4 &v) {
    const uint64_t lo = (uint64_t)v.x | (uint64_t)v.y << 32, hi = (uint64_t)v.z | (uint64_t)v.w << 32;
    asm volatile("{\n\t.reg .b128 v;\n\tmov.b128 v, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], v;\n\t}\n" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ void post16(float *p, float a, float b, float c, float d) {   // (the first word of a piece tells: never all ones)
    post16(p, make_uint4(min(__float_as_uint(a), 0xfffffffeu), __float_as_uint(b), __float_as_uint(c), __float_as_uint(d)));
}
__device__ __forceinline__ float4 as_f4(const uint4 &v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ void unpack8(const uint4 &q, float (&f)[8]) {
    const float2 a = unpack_h2(q.x), b = unpack_h2(q.y), c = unpack_h2(q.z), d = unpack_h2(q.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
    f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_h2(f[0], f[1]), pack_h2(f[2], f[3]), pack_h2(f[4], f[5]), pack_h2(f[6], f[7]));
}
// f16 of the values of lanes l .. l + 7, for lanes that are a multiple of 8
__device__ __forceinline__ uint4 gather8(float v) {
    const uint32_t u = __half_as_ushort(__float2half_rn(v)), w = u | __shfl_down_sync(0xffffffffu, u, 1) << 16;
    return make_uint4(w, __shfl_down_sync(0xffffffffu, w, 2), __shfl_down_sync(0xffffffffu, w, 4), __shfl_down_sync(0xffffffffu, w, 6));
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

// acc += a step's product: 16 weight rows (a: byte of this lane's row g of the tile in w, rb8: eight rows on) times 128 k (unit u) of
// the activations, x: this lane's k = 8t .. + 7 of column g, 32 apart.
__device__ __forceinline__ void step_mma(float (&acc)[4], const uint8_t *w, uint32_t a, uint32_t rb8, int u, int t, const uint4 *x, bool col) {
    uint32_t cw[2][2];
    float d[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t b = a + (h ? rb8 : 0u) + (uint32_t)((u >> 1) * 66);
        lds_codes<2>(w, b + (uint32_t)(32 * (u & 1) + 8 * t), cw[h]);
        d[h] = __half2float(__ushort_as_half((unsigned short)lds16(w, b + 64u))) * 512.0f;
    }
    float c[2][4] = {};
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const uint4 v = col ? x[4 * l] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int q = 0; q < 2; q++)
            sm_mma(c[q], codes_f16<2, 1>(cw[0][q], l), codes_f16<2, 1>(cw[1][q], l), codes_f16<2, 1>(cw[0][q] >> 8, l), codes_f16<2, 1>(cw[1][q] >> 8, l),
                   q ? v.z : v.x, q ? v.w : v.y);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i] = fmaf(c[0][i] + c[1][i], d[i >> 1], acc[i]);
}
__device__ __forceinline__ void put_sums(float *red, float (&acc)[4], int g, int t) {
    float *dst = red + 2 * t * RED_COL + g;
    dst[0] = acc[0];
    dst[RED_COL] = acc[1];
    dst[8] = acc[2];
    dst[RED_COL + 8] = acc[3];
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
}
// Two lanes (16 apart) add up to 16 warps' sums of one element.
__device__ __forceinline__ float sum_parts(const float *src, int n, int lane) {
    const int first = lane >> 4;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = first + 2 * j < n ? src[(first + 2 * j) * RED_PART] : 0.f;
    const float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    return s + __shfl_xor_sync(0xffffffffu, s, 16);
}

// The norms between two phases, 1 << row_log threads per row: resid = f16(rms_norm(y, w1) + resid) unless y is NULL, then
// f16(rms_norm(resid, w2)) to dst.  NJ: 16-byte pieces of a row per thread.  False: a wait ran out (all threads).
template <int NJ, typename Here>
__device__ __forceinline__ bool norm_rows(int m, int pieces, float eps, const uint4 *y, const uint4 *w1, uint4 *resid, const uint4 *w2, uint4 *dst, int dst_stride,
                                          float *sh, int tid, int row_log, uint32_t limit, bool late, Here &&here) {
    const int lane = tid & 31, warp = tid >> 5, row = tid >> row_log, at = tid & ((1 << row_log) - 1), wpr = 1 << (row_log - 5);
    const bool act = row < m;
    auto row_sum = [&](float s, float *sh_, bool fail, bool &any) -> float {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sh_[warp] = s;
        any = wide_sync_or(fail);
        s = lane < wpr ? sh_[row * wpr + lane] : 0.f;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return __shfl_sync(0xffffffffu, s, 0);
    };
    uint4 r[NJ];
    bool any;
    uint4 *res = resid + row * pieces;
    if (y) {
        const uint4 *src = y + row * pieces;
        bool fail;
        uint32_t tries = 0;
#pragma unroll 1
        do {
            fail = false;
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int c = at + (j << row_log);
                r[j] = make_uint4(0u, 0u, 0u, 0u);
                if (act && c < pieces) r[j] = take16(src + c);
            }
#pragma unroll
            for (int j = 0; j < NJ; j++) fail = fail || !here(r[j]);
        } while (fail && ++tries < limit);
        __syncwarp();
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            float x[8];
            unpack8(r[j], x);
#pragma unroll
            for (int e = 0; e < 8; e++) s = fmaf(x[e], x[e], s);
        }
        const float rms = rsqrtf(row_sum(s, sh, fail || late, any) / (float)(8 * pieces) + eps);
        if (any) return false;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int c = at + (j << row_log);
            if (act && c < pieces) {
                float x[8], a[8], v[8];
                unpack8(r[j], x);
                unpack8(w1[c], a);
                unpack8(res[c], v);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = x[e] * rms * a[e] + v[e];
                res[c] = r[j] = pack8(v);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int c = at + (j << row_log);
            r[j] = act && c < pieces ? res[c] : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        float x[8];
        unpack8(r[j], x);
#pragma unroll
        for (int e = 0; e < 8; e++) s = fmaf(x[e], x[e], s);
    }
    const float rms = rsqrtf(row_sum(s, sh + ST_NW, late, any) / (float)(8 * pieces) + eps);
    if (any) return false;
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int c = at + (j << row_log);
        if (act && c < pieces) {
            float x[8], a[8];
            unpack8(r[j], x);
            unpack8(w2[c], a);
#pragma unroll
            for (int e = 0; e < 8; e++) x[e] = x[e] * rms * a[e];
            dst[row * dst_stride + c] = pack8(x);
        }
    }
    return true;
}

template <int BITS>
__global__ void __launch_bounds__(ST_NT + 32, 1) step_layers_kernel(const __grid_constant__ LcStepParams p) {
    using C = AttnCfg<HD, BITS>;
    using W = Wide<C>;
    constexpr int KB = W::KB, CB = C::CB, NLEV = 1 << BITS, STAGES = stages_of(BITS);
    static_assert(W::NT == ST_NT, "one block shape");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[4];          // regions A and B: filled, free again
    __shared__ float sh_red[2 * ST_NW];
    __shared__ float l_s[ST_NW * G];
    __shared__ uint32_t pos_s[LC_STEP_MAX_LANES], mail_s[8];   // mail_s: where a layer's exchange buffers begin, bytes (Q_M ..)
    __shared__ uint8_t tile_s[2][MAX_TILES][2];        // first warp on a tile of Q/K/V (0) or gate/up (1), and how many
    __shared__ int4 share_s[2][ST_NW];                 // a warp's steps there: from, to, the first one's tile and unit
    __shared__ __align__(16) LcStepLayer layer_s[3];   // the layer at hand, the one before and the one after (layer mod 3)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int cta = blockIdx.x, ctas = gridDim.x;
    const int H = p.hidden, m = p.m, n_q = p.n_q, n_kv = p.n_kv;
    uint2 *lut = reinterpret_cast<uint2 *>(smem);
    uint4 *frag_s = reinterpret_cast<uint4 *>(smem + C::LUT_BYTES);                        // query fragments of an item
    float *sg_s = reinterpret_cast<float *>(smem + C::LUT_BYTES + C::Q_BYTES);             // signs
    uint8_t *wa_s = smem + C::LUT_BYTES + C::Q_BYTES + HD * 4, *wb_s = smem + p.off_b;     // norm weights and weights of Q/K/V or gate/up; of O or down
    uint8_t *work = smem + p.off_u;                                                        // one phase's work space
    float2 *rot_s = reinterpret_cast<float2 *>(smem + p.off_rot);                          // [m][128] cos, sin
    uint4 *resid = reinterpret_cast<uint4 *>(smem + p.off_resid);                          // [m][H] halves
    uint4 *xs = reinterpret_cast<uint4 *>(work);                                           // a phase's activations, rows xs_row pieces apart
    float *red = reinterpret_cast<float *>(work + p.off_red);                              // [warp + tile]: sums (put_sums)
    const uint32_t bar_a = smem_u32(&bars[0]), bar_b = smem_u32(&bars[1]), free_a = smem_u32(&bars[2]), free_b = smem_u32(&bars[3]);

    // ---- tiles of 16 weight rows: CTA c has [T c / ctas, T (c + 1) / ctas) of a phase's T ----
    auto tile_of = [&](int T, int c) -> int { return T * c / ctas; };
    const int qd = n_q * HD, kd = n_kv * HD;
    const int t_qkv = (qd + 2 * kd) / 16, t_gate = p.inter / 8, t_out = H / 16;
    const int rb_h = H / 256 * 66, rb_q = n_q * 66, rb_i = p.inter / 256 * 66;   // bytes of a weight row
    const int a0[2] = {tile_of(t_qkv, cta), tile_of(t_gate, cta)};
    const int an[2] = {tile_of(t_qkv, cta + 1) - a0[0], tile_of(t_gate, cta + 1) - a0[1]};
    const int b0 = tile_of(t_out, cta), bn = tile_of(t_out, cta + 1) - b0;       // (at most one tile)
    uint32_t par_a = 0, par_b = 0;
    const int halves = 2 * p.n_layers;
    if (tid == 0)
        for (int i = 0; i < 4; i++) mbar_init(smem_u32(&bars[i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    auto fetch_layer = [&](int l) {
        static_assert(sizeof(LcStepLayer) % 8 == 0 && sizeof(LcStepLayer) <= 256, "copied by a warp in 8-byte words");
        if (l < p.n_layers && lane < (int)(sizeof(LcStepLayer) / 8))
            reinterpret_cast<uint64_t *>(&layer_s[l % 3])[lane] = reinterpret_cast<const uint64_t *>(&p.layer[l])[lane];
    };
    if (warp == ST_NW) {
        fetch_layer(0);
        fetch_layer(1);
    }
    if (tid < m) pos_s[tid] = p.positions[tid];
    if (tid == 0) {
        const uint32_t mq = 2u * m * qd, mk = 2u * m * kd, mh = 2u * m * H;
        uint32_t at = COUNTS;
        mail_s[Q_M] = at;
        mail_s[K_M] = at += mq;
        mail_s[V_M] = at += mk;
        mail_s[ATTN_M] = at += mk;
        mail_s[O_M] = at += mq;
        mail_s[DOWN_M] = at += mh;
        mail_s[GATE_M] = at += mh;
        mail_s[PART_M] = at + 2u * m * p.inter;
    }
    __syncthreads();
    if (warp == ST_NW) {
        // ---- the fetching warp.  Region A of half-layer h: the norm weights w1 and w2 (h == 0 has no first norm), then the tiles; region B the
        //      tile of O or down.  A region is fetched anew as soon as its readers are done with it. ----
#pragma unroll 1
        for (int h = 0;; h++) {
            const int ffn = h & 1, n = h < halves ? an[ffn] : 0, rows = ffn ? 8 : 16, pieces = ffn ? 2 * n : n;
            const LcStepLayer &L = layer_s[(h >> 1) % 3], &before = layer_s[((h >> 1) + 2) % 3];
            if (h > 0 && !mbar_wait_warp(free_a, (uint32_t)(h - 1) & 1u, p.wait_limit)) break;   // (expired)
            if (lane == 0) mbar_arrive_expect_tx(bar_a, (uint32_t)(n * 16 * rb_h + (h > 0 ? 4 : 2) * H));
            __syncwarp();
            const uint32_t dst = smem_u32(wa_s);
#pragma unroll 1
            for (int i = lane - 2; i < pieces; i += 32) {
                const void *src;
                uint32_t bytes = (uint32_t)(rows * rb_h), off = (uint32_t)(4 * H + i * rows * rb_h);
                if (i < 0) {
                    if (i == -2) src = ffn ? L.post_attn_norm : before.post_ffn_norm;
                    else src = h == halves ? p.final_norm : (ffn ? L.ffn_norm : L.attn_norm);
                    bytes = 2 * H;
                    off = (uint32_t)(i + 2) * 2 * H;
                    if (i == -2 && h == 0) continue;
                } else if (ffn) {
                    src = ((i & 1) ? L.wup : L.wgate) + (size_t)(a0[1] + (i >> 1)) * 8 * rb_h;
                } else {
                    int r = (a0[0] + i) * 16;
                    const uint8_t *wm = L.wq;
                    if (r >= qd + kd) { r -= qd + kd; wm = L.wv; }
                    else if (r >= qd) { r -= qd; wm = L.wk; }
                    src = wm + (size_t)r * rb_h;
                }
                bulk_g2s(dst + off, src, bytes, bar_a);
            }
            __syncwarp();
            if (h < halves && bn > 0) {
                if (h > 0 && !mbar_wait_warp(free_b, (uint32_t)(h - 1) & 1u, p.wait_limit)) break;   // (expired)
                if (lane == 0) {
                    const uint32_t bytes = (uint32_t)(16 * (ffn ? rb_i : rb_q));
                    mbar_arrive_expect_tx(bar_b, bytes);
                    bulk_g2s(smem_u32(wb_s), (ffn ? L.wdown : L.wo) + (size_t)b0 * bytes, bytes, bar_b);
                }
            }
            if (ffn) fetch_layer((h >> 1) + 2);   // (into the place of the layer before, whose last reader has freed region A)
            __syncwarp();
            if (h == (cta == 0 ? halves : halves - 1)) return;
        }
        tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, lane);
        return;
    }
    auto weights = [&](uint32_t bar, uint32_t parity) -> bool { return mbar_wait_warp(bar, parity, p.wait_limit); };
    auto here = [&](const uint4 &v) -> bool { return v.x != 0xffffffffu && !p.never; };

    // ---- once: table of levels, signs, rotations of every lane's position, embedding rows ----
    const float gamma = attn_table<C, ST_NW>(p.levels, lut, lane, warp, [] { wide_sync(); });
    const uint2 *lut_lane = lut + (lane & (LUT_COPIES - 1));
    if (tid < HD) sg_s[tid] = p.signs[tid];
#pragma unroll 1
    for (int i = tid; i < m * 128; i += ST_NT) {
        const float freq = 1.0f / powf(p.theta, (float)(2 * (i & 127)) / (float)HD), ang = (float)pos_s[i >> 7] * freq;
        rot_s[i] = make_float2(cosf(ang), sinf(ang));
    }
#pragma unroll 1
    for (int i = tid; i < m * H; i += ST_NT) {
        const int r = i / H, e = i - r * H, j = e & 31;
        const uint8_t *q = p.embed + (size_t)p.tokens[r] * (size_t)(H / 32 * 18) + (e >> 5) * 18;
        const float d = __half2float(*reinterpret_cast<const __half *>(q));
        const unsigned byte = q[2 + (j & 15)], qv = j < 16 ? (byte & 15u) : (byte >> 4);
        __half v = __float2half_rn(((float)qv - 8.0f) * d);
        if (p.embed_scale != 1.0f) v = __float2half_rn(__half2float(v) * p.embed_scale);
        reinterpret_cast<__half *>(resid)[i] = v;
    }
    wide_sync();

    // The weight steps of a phase, a tile of 16 rows times a unit of 128 k each: the warps share the steps of a CTA evenly, tile after
    // tile.  A phase with fewer steps than warps occupies the first ones.
    const int units_h = H / UNIT;
    auto share = [&](int total, int w) -> int { const int on = min(total, ST_NW); return w < on ? total * w / on : total; };
    if (tid < 2 * ST_NW) {
        const int ffn = tid / ST_NW, w = tid % ST_NW, total = an[ffn] * units_h, i = share(total, w);
        share_s[ffn][w] = make_int4(i, share(total, w + 1), i / units_h, i % units_h);
    }
    if (tid < 2 * MAX_TILES) {
        const int ffn = tid / MAX_TILES, tile = tid % MAX_TILES, total = an[ffn] * units_h, on = min(total, ST_NW);
        if (tile < an[ffn]) {
            const int first = ((tile * units_h + 1) * on - 1) / total, last = ((tile + 1) * units_h * on - 1) / total;   // (the last w whose share begins there or before)
            tile_s[ffn][tile][0] = (uint8_t)first;
            tile_s[ffn][tile][1] = (uint8_t)(last - first + 1);
        }
    }
    wide_sync();
    // threads of a row in the norms
    const int row_log = m <= 2 ? 8 : 7;
    const int inv_m = (65536 + m - 1) / m;   // (i * inv_m >> 16 is i / m for i below 128)

#pragma unroll 1
    for (int h = 0;; h++) {
        const int layer = h >> 1, ffn = h & 1;
        if (h == halves && cta != 0) return;   // (the final norm is one CTA's)
        const LcStepLayer &L = layer_s[layer % 3];
        uint8_t *mail = p.mail + (h < halves ? L.mail : 0);
        auto rows_at = [&](int which) -> __half * { return reinterpret_cast<__half *>(mail + mail_s[which]); };
        // Two projections: Q, K, V or gate and up on the normed rows, O or down on what attention or the gate made of them.
#pragma unroll 1
        for (int second = 0; second < 2; second++) {
        if (second && !ffn) {
            // ---- attention: item (lane, 8 heads, split); the last split is the newest key alone ----
            const int nch = n_q / 8, gch = nch / n_kv, S = (int)L.splits, items = m * nch * (S + 1);
            struct Range { uint32_t pos, begin, old_keys, per; bool newest; };
            auto range_of = [&](int li) -> Range {
                Range r;
                r.pos = pos_s[li];
                r.newest = L.ring != 0u || r.pos < L.lane_rows;
                const uint32_t end = r.newest ? r.pos : L.lane_rows;   // (a position past the lane's rows is clamped and reported)
                r.begin = L.window > 0u && r.pos + 1u > L.window ? r.pos + 1u - L.window : 0u;
                r.old_keys = end > r.begin ? end - r.begin : 0u;
                auto keys_of = [&](uint32_t n) -> uint32_t { return max(((r.old_keys + n - 1u) / n + (KB - 1)) & ~(uint32_t)(KB - 1), (uint32_t)KB); };
                r.per = keys_of(min((uint32_t)S, (uint32_t)FEW_SPLITS));
                if (r.per > FULL_SPLIT * KB) r.per = max(keys_of((uint32_t)S), (uint32_t)(FULL_SPLIT * KB));   // (long ones: all the splits)
                return r;
            };
            uint8_t *scratch = work + STAGES * W::STAGE;
            float *norm_s = reinterpret_cast<float *>(scratch + W::PART_BYTES + W::P_BYTES + ST_NW * G * 4);   // [2][2 KB]
            uint32_t *normw_s = reinterpret_cast<uint32_t *>(norm_s + 4 * KB);                                                     // [STAGES][2 KB]
#pragma unroll 1
            for (int it = cta; it < items; it += ctas) {
                const int r8 = it / (S + 1), s = it - r8 * (S + 1), li = r8 / nch, hc = r8 - li * nch, kvh = hc / gch;
                const Range R = range_of(li);
                const bool newest = s == S;
                const uint32_t k_begin = newest ? R.pos : R.begin + (uint32_t)s * R.per;
                const uint32_t k_end = newest ? (R.newest ? R.pos + 1u : R.pos) : min(R.begin + R.old_keys, k_begin + R.per);
                const int blocks = k_end > k_begin ? (int)((k_end - k_begin + KB - 1) / KB) : 0;
                auto slot_of = [&](uint32_t key) -> size_t { return ((size_t)li * L.lane_rows + (L.ring ? key % L.ring : key)) * n_kv + kvh; };
                if (newest && !R.newest && tid == 0) atomicExch(p.status, LC_DEV_STATUS_POSITION);
                if (blocks == 0) continue;
                WideAcc<C> acc;
                acc.clear();
                uint4 bq[2];
                uint32_t odd = 0;   // whether this thread's norm of a block is the upper half of its word, a bit per stage
                // Round r fetches block r (the keys of earlier steps do not depend on this one: the first ones ahead of the query)
                // and works on block r - ahead.
                const int ahead = newest ? 0 : min(blocks, STAGES - 1);
#pragma unroll 1
                for (int r = 0; r < blocks + ahead; r++) {
                    const int blk = r - ahead;
                    if (!newest && blk >= 0) {
                        if (ahead == STAGES - 1) cp_async_wait<STAGES - 2>();
                        else cp_async_wait<0>();
                        if (tid < 2 * KB) {
                            const uint32_t wd = normw_s[blk % STAGES * 2 * KB + tid];
                            const float n = __half2float(__ushort_as_half((unsigned short)(odd >> (blk % STAGES) & 1u ? wd >> 16 : wd)));
                            norm_s[(blk & 1) * 2 * KB + tid] = (int)(k_end - k_begin) - blk * KB > (tid & (KB - 1)) ? n * gamma : 0.f;
                        }
                    }
                    if (blk == 0) {
                        // rows: warp w < 8 the query of head w; for the newest key warp 8 its row of K, warp 9 of V.  Norm, rotary embedding,
                        // rotation; then a query is split into fragments and a row of the cache into codes.
                        bool fail = false;
                        if (warp < (newest ? 10 : 8)) {
                            const bool query = warp < 8, value = warp == 9;
                            const __half *src = rows_at(query ? Q_M : (value ? V_M : K_M)) + (query ? li * n_q + hc * 8 + warp : li * n_kv + kvh) * HD;
                            float x[8], w[8], sg[8], cs[8], sn[8];
                            unpack8(__ldg(reinterpret_cast<const uint4 *>(query ? L.q_norm : L.k_norm) + lane), w);
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const float2 a = rot_s[li * 128 + ((8 * lane + e) & 127)];
                                cs[e] = value ? 1.f : a.x;
                                sn[e] = value ? 0.f : a.y;
                                w[e] = value ? 1.f : w[e];
                                sg[e] = sg_s[8 * lane + e];
                            }
                            uint4 raw;
                            uint32_t tries = 0;
#pragma unroll 1
                            do {
                                raw = take16(src + 8 * lane);
                                fail = !here(raw);
                            } while (fail && ++tries < p.wait_limit);
                            __syncwarp();
                            unpack8(raw, x);
                            warp_head_norm(x, w, p.eps);
                            warp_rope(x, cs, sn, HD / 2, lane);
                            float norm = 1.f;
                            if (!query) {   // TurboQuant::encode_into
                                float *sq = reinterpret_cast<float *>(scratch) + (warp - 8) * HD;
#pragma unroll
                                for (int e = 0; e < 8; e++) sq[8 * lane + e] = __fmul_rn(x[e], x[e]);
                                __syncwarp();
                                if (lane == 0) norm = sequential_norm<HD>(sq);
                                norm = __shfl_sync(0xffffffffu, norm, 0);
                                const float inv = norm > 0.f ? __fdiv_rn(1.0f, norm) : 1.f;
#pragma unroll
                                for (int e = 0; e < 8; e++) x[e] = __fmul_rn(x[e], inv);
                            }
#pragma unroll
                            for (int e = 0; e < 8; e++) x[e] = __fmul_rn(x[e], sg[e]);
                            fwht_warp_row<8>(x, lane);
                            const float k = __fdiv_rn(query ? p.softmax_scale : 1.0f, __fsqrt_rn((float)HD));
#pragma unroll
                            for (int e = 0; e < 8; e++) x[e] = __fmul_rn(x[e], k);
                            if (query) {
                                uint4 f[2];
                                split_h2(x[0], x[1], f[0].x, f[0].z);
                                split_h2(x[2], x[3], f[0].y, f[0].w);
                                split_h2(x[4], x[5], f[1].x, f[1].z);
                                split_h2(x[6], x[7], f[1].y, f[1].w);
                                uint4 *dst = frag_s + ((lane >> 2) * 32 + 4 * warp + (lane & 3)) * 2;   // (part lane >> 2 contracts over these dims)
                                dst[0] = f[0];
                                dst[1] = f[1];
                            } else {
                                unsigned codes = 0;   // (8 * BITS <= 32)
                                float lv[NLEV];
#pragma unroll
                                for (int i = 0; i < NLEV; i++) lv[i] = __ldg(p.levels + i);
#pragma unroll
                                for (int e = 0; e < 8; e++) {
                                    unsigned best = 0;
                                    float bd = INFINITY;
#pragma unroll
                                    for (int j = 0; j < NLEV; j++) {
                                        const float dd = fabsf(__fsub_rn(x[e], lv[j]));
                                        if (dd < bd) { bd = dd; best = (unsigned)j; }
                                    }
                                    codes |= best << (BITS * e);
                                }
                                const __half nh = __float2half_rn(norm);
                                store_warp_codes<HD, BITS>(codes, lane, work + (value ? KB * W::RS : 0));
                                for (int i = lane; i < KB; i += 32) norm_s[(value ? KB : 0) + i] = i == 0 ? __half2float(nh) * gamma : 0.f;
                                if (hc == kvh * gch && !__any_sync(0xffffffffu, fail)) {
                                    const size_t sl = slot_of(R.pos);
                                    store_warp_codes<HD, BITS>(codes, lane, (value ? L.v_codes : L.k_codes) + sl * CB);
                                    if (lane == 0) (value ? L.v_norms : L.k_norms)[sl] = nh;
                                }
                            }
                        }
                        if (wide_sync_or(fail)) goto expired;
                        bq[0] = frag_s[((warp & 7) * 32 + lane) * 2];
                        bq[1] = frag_s[((warp & 7) * 32 + lane) * 2 + 1];
                    } else if (blk > 0) {
                        wide_sync();   // block and norms are in place; everybody is done with the block before
                    }
                    if (!newest) {
                        if (r < blocks) {
                            constexpr int CPR = CB / 16;
                            const uint32_t dst = smem_u32(work) + (uint32_t)(r % STAGES) * W::STAGE, t0 = k_begin + (uint32_t)r * KB;
#pragma unroll 1
                            for (int i = tid; i < 2 * KB * CPR; i += ST_NT) {   // K rows, then V rows
                                const uint32_t row = (uint32_t)i / CPR, off = ((uint32_t)i - row * CPR) * 16u;
                                const size_t sl = slot_of(min(t0 + (row & (KB - 1)), k_end - 1u));   // (past the end: the last key's)
                                cp_async16(dst + row * W::RS + off, (row < KB ? L.k_codes : L.v_codes) + sl * CB + off);
                            }
                            if (tid < 2 * KB) {   // K's norms, then V's: the word that holds each
                                const size_t sl = slot_of(min(t0 + (uint32_t)(tid & (KB - 1)), k_end - 1u));
                                cp_async4(smem_u32(normw_s + r % STAGES * 2 * KB + tid), (tid < KB ? L.k_norms : L.v_norms) + (sl & ~(size_t)1));
                                odd = (odd & ~(1u << (r % STAGES))) | (uint32_t)(sl & 1) << (r % STAGES);
                            }
                        }
                        cp_async_commit();
                    }
                    if (blk >= 0)
                        wide_block<C>(acc, work + (blk % STAGES) * W::STAGE, norm_s + (blk & 1) * 2 * KB, (int)(k_end - k_begin) - blk * KB, bq, lut_lane,
                                      scratch, tid);
                }
                // the split's sums, unnormalised: the warps of the second half of the keys hand theirs over
                float *part = reinterpret_cast<float *>(mail + mail_s[PART_M]) + ((size_t)r8 * (S + 1) + s) * 8 * PROW;
                float l = acc.l;
                l += __shfl_xor_sync(0xffffffffu, l, 8);
                l += __shfl_xor_sync(0xffffffffu, l, 16);
                if (lane < G) l_s[warp * G + lane] = l;
                float4 *half_s = reinterpret_cast<float4 *>(scratch);
                if (warp >= 8) {
                    half_s[(warp - 8) * 64 + lane] = make_float4(acc.o[0][0], acc.o[0][2], acc.o[1][0], acc.o[1][2]);
                    half_s[(warp - 8) * 64 + 32 + lane] = make_float4(acc.o[0][1], acc.o[0][3], acc.o[1][1], acc.o[1][3]);
                }
                wide_sync();
                if (warp < 8) {
                    const float4 a = half_s[warp * 64 + lane], b = half_s[warp * 64 + 32 + lane];
                    float *dst = part + (2 * t) * PROW + 4 + 32 * warp + 4 * g;
                    post16(dst, acc.o[0][0] + a.x, acc.o[0][2] + a.y, acc.o[1][0] + a.z, acc.o[1][2] + a.w);
                    post16(dst + PROW, acc.o[0][1] + b.x, acc.o[0][3] + b.y, acc.o[1][1] + b.z, acc.o[1][3] + b.w);
                } else if (warp == 8 && lane < G) {
                    l = 0.f;
#pragma unroll
                    for (int w = 0; w < ST_NW; w++) l += l_s[w * G + lane];
                    post16(part + lane * PROW, acc.m, l, 0.f, 0.f);
                }
                wide_sync();   // (the work space is written again)
            }
            // ---- merge of the splits: one head of one lane per CTA (from the last CTA down), 64 threads of four dims for every eighth split ----
#pragma unroll 1
            for (int e = ctas - 1 - cta; e < m * n_q; e += ctas) {
                const int li = e / n_q, head = e - li * n_q, grp = tid >> 6, d4 = tid & 63;
                const Range R = range_of(li);
                const int n_old = (int)((R.old_keys + R.per - 1u) / R.per), n = n_old + (R.newest ? 1 : 0);
                const float *part = reinterpret_cast<const float *>(mail + mail_s[PART_M]) + ((size_t)(li * nch + head / 8) * (S + 1) * 8 + (head & 7)) * PROW;
                auto at = [&](int j) -> const float * { return part + (size_t)(j < n_old ? j : S) * 8 * PROW; };
                float m_run = -INFINITY, l_run = 0.f;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
                constexpr int AT_ONCE = 4;   // splits whose trips pass together
                uint32_t tries = 0;
#pragma unroll 1
                for (int j0 = grp; j0 < n; j0 += 8 * AT_ONCE) {
                    uint4 ml[AT_ONCE], v[AT_ONCE];
                    bool fail;
#pragma unroll 1
                    do {
                        fail = false;
#pragma unroll
                        for (int u = 0; u < AT_ONCE; u++) {
                            const float *src = at(min(j0 + 8 * u, n - 1));
                            ml[u] = take16(src);
                            v[u] = take16(src + 4 + 4 * d4);
                        }
#pragma unroll
                        for (int u = 0; u < AT_ONCE; u++) fail = fail || !(here(ml[u]) && here(v[u]));
                    } while (fail && ++tries < p.wait_limit);
#pragma unroll
                    for (int u = 0; u < AT_ONCE; u++) {
                        if (j0 + 8 * u >= n) break;
                        const float4 x = as_f4(v[u]);
                        const float mj = __uint_as_float(ml[u].x), lj = __uint_as_float(ml[u].y);
                        const float m_new = fmaxf(m_run, mj), f0 = m_run == -INFINITY ? 0.f : expf(m_run - m_new), f1 = mj == -INFINITY ? 0.f : expf(mj - m_new);
                        a.x = a.x * f0 + x.x * f1; a.y = a.y * f0 + x.y * f1; a.z = a.z * f0 + x.z * f1; a.w = a.w * f0 + x.w * f1;
                        l_run = l_run * f0 + lj * f1;
                        m_run = m_new;
                    }
                }
                float *grp_s = reinterpret_cast<float *>(work);   // [8]: {max, sum, -, -}, 256 sums; then room for the transform
                *reinterpret_cast<float4 *>(grp_s + grp * PROW + 4 + 4 * d4) = a;
                if (d4 == 0) *reinterpret_cast<float2 *>(grp_s + grp * PROW) = make_float2(m_run, l_run);
                if (wide_sync_or(tries >= p.wait_limit)) goto expired;
                float gmax = -INFINITY, gsum = 0.f, x = 0.f;
                const int d = tid & (HD - 1);   // (both halves of the CTA do the same)
#pragma unroll
                for (int i = 0; i < 8; i++) gmax = fmaxf(gmax, grp_s[i * PROW]);
#pragma unroll 1
                for (int i = 0; i < min(n, 8); i++) {
                    const float f = expf(grp_s[i * PROW] - gmax);
                    gsum += f * grp_s[i * PROW + 1];
                    x += f * grp_s[i * PROW + 4 + d];
                }
                x = gsum > 0.f ? x / gsum : 0.f;
                #pragma unroll 1
                for (unsigned len = 1; len < 32; len <<= 1) {
                    const float o = __shfl_xor_sync(0xffffffffu, x, len);
                    x = (tid & len) ? o - x : x + o;
                }
                x = lc_fwht_cross_warp<8>(x, grp_s + 8 * PROW, tid, [] { wide_sync(); });
                const uint4 piece = gather8(x * (1.0f / sqrtf((float)HD)) * sg_s[d]);
                if (tid < HD && (lane & 7) == 0) post16(rows_at(ATTN_M) + e * HD + d, piece);
                wide_sync();
            }
        }
        const int n = second ? bn : (h < halves ? an[ffn] : 0);
        const int K = second ? (ffn ? p.inter : qd) : H, units = K / UNIT;
        const int xs_row = units * (UNIT / 8) + 4, rb = K / 256 * 66;
        const uint8_t *w = second ? wb_s : wa_s + 4 * H;
        if (second && n == 0) break;
        const bool late = !weights(second ? bar_b : bar_a, second ? par_b : par_a);   // (as a rule long there)
        if (second) par_b ^= 1u;
        else par_a ^= 1u;
        {
            if (second) {
                const uint4 *src = reinterpret_cast<const uint4 *>(rows_at(ffn ? GATE_M : ATTN_M));
                const int row_pieces = units * (UNIT / 8), row = tid >> row_log, step = 1 << row_log;
                bool fail = false;
#pragma unroll 1
                for (int i0 = tid & (step - 1); row < m && i0 < row_pieces && !fail; i0 += 3 * step) {
                    uint4 v[3];
                    uint32_t tries = 0;
#pragma unroll 1
                    do {
                        fail = false;
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            v[j] = make_uint4(0u, 0u, 0u, 0u);
                            if (i0 + j * step < row_pieces) v[j] = take16(src + (size_t)row * (K / 8) + i0 + j * step);
                        }
#pragma unroll
                        for (int j = 0; j < 3; j++) fail = fail || !here(v[j]);
                    } while (fail && ++tries < p.wait_limit);
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        if (i0 + j * step < row_pieces) xs[row * xs_row + i0 + j * step] = v[j];
                }
                __syncwarp();
                if (wide_sync_or(fail || late)) goto expired;
            } else {
                const bool last = h == halves;
                const uint4 *y = h == 0 ? nullptr
                                        : reinterpret_cast<const uint4 *>(p.mail + layer_s[ffn ? layer % 3 : (layer + 2) % 3].mail + mail_s[ffn ? O_M : DOWN_M]);
                const uint4 *w1 = reinterpret_cast<const uint4 *>(wa_s), *w2 = w1 + H / 8;
                uint4 *dst = last ? reinterpret_cast<uint4 *>(p.normed) : xs;
                const int stride = last ? H / 8 : xs_row;
                if (y) {
                    // Every CTA reads these rows.  Until they are nearly all there only one thread asks, for the count of the posts (begun at -1; a
                    // hint: it says nothing about the data): the readers' traffic on the rows' lines delays the posts (898 -> 870 us a step of one
                    // lane; for the rows of attention and of the gate, which fewer CTAs read, asking first costs more than it saves).
                    if (tid == 0) {
                        const uint8_t *count = p.mail + layer_s[ffn ? layer % 3 : (layer + 2) % 3].mail + (ffn ? 0 : 128);
                        uint32_t c, tries = 0;
#pragma unroll 1
                        do {
                            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(c) : "l"(count) : "memory");
                        } while (c + 1 < (uint32_t)(t_out * m) && ++tries < p.wait_limit);
                    }
                    wide_sync();
                }
                const bool ok = m <= 2 ? norm_rows<1>(m, H / 8, p.eps, y, w1, resid, w2, dst, stride, sh_red, tid, row_log, p.wait_limit, late, here)
                              : norm_rows<2>(m, H / 8, p.eps, y, w1, resid, w2, dst, stride, sh_red, tid, row_log, p.wait_limit, late, here);
                if (!ok) goto expired;
                if (last) return;
                wide_sync();
            }
            const int4 mine = second ? make_int4(units * warp / ST_NW, units * (warp + 1) / ST_NW, 0, units * warp / ST_NW) : share_s[ffn][warp];
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            int i = mine.x, tile = mine.z, u = mine.w;
            const int end = mine.y;
#pragma unroll 1
            for (; i < end; i++) {
                step_mma(acc, w, (uint32_t)((tile * 16 + g) * rb), (uint32_t)(8 * rb), u, t, xs + g * xs_row + u * (UNIT / 8) + t, g < m);
                u++;
                if (!second && (u == units || i + 1 == end)) {
                    put_sums(red + (warp + tile) * RED_PART, acc, g, t);   // (no two (warp, tile) of a share have one sum)
                    tile++;
                    u = 0;
                }
            }
            if (second) put_sums(red + warp * RED_PART, acc, g, t);
        }
        wide_sync();
        if (tid == 0) mbar_arrive(second ? free_b : free_a);
        {
            const bool gate = ffn && !second;
            // A warp makes 16 rows of a column, a tile's or of gate * up two tiles', and posts them together: consumers are reading all along,
            // and every write into a line has to pass between their reads (16-byte posts by a warp each: a step took 10 % longer).
            const int groups = gate ? (n + 1) >> 1 : n, row = lane & 15;
#pragma unroll 1
            for (int pc = warp; pc < groups * m; pc += ST_NW) {
                const int gr = (pc * inv_m) >> 16, col = pc - gr * m, tl = gate ? 2 * gr + (row >> 3) : gr;
                const bool there = tl < n;
                const int parts = second ? ST_NW : (there ? tile_s[ffn][tl][1] : 0), from = second || !there ? 0 : tile_s[ffn][tl][0] + tl;
                const float *src = red + from * RED_PART + col * RED_COL + (gate ? row & 7 : row);
                float v = sum_parts(src, parts, lane);
                if (gate) v = geglu_f(v, sum_parts(src + 8, parts, lane));
                const uint4 piece = gather8(v);
                if (there && (lane == 0 || lane == 8)) {
                    __half *dst;
                    if (second) {
                        dst = rows_at(ffn ? DOWN_M : O_M) + col * H + b0 * 16;
                    } else if (gate) {
                        dst = rows_at(GATE_M) + col * p.inter + (a0[1] + 2 * gr) * 8;
                    } else {
                        const int r = (a0[0] + tl) * 16, which = r < qd ? Q_M : (r < qd + kd ? K_M : V_M);
                        dst = rows_at(which) + (which == Q_M ? col * qd + r : col * kd + r - qd - (which == V_M ? kd : 0));
                    }
                    post16(dst + lane, piece);
                    if (second && lane == 0)
                        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;\n" ::"l"(mail + (ffn ? 128 : 0)) : "memory");
                }
            }
        }
        wide_sync();   // (the work space is written again)
        }
    }
expired:   // a wait ran out: this CTA leaves, and the waits of the others run out, too
    tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, tid);
}

int cdiv(int a, int b) { return (a + b - 1) / b; }

// Blocks of 64 keys that a layer's attention reads of a lane at most.
int blocks_of(uint32_t window, uint32_t lane_rows) { return (int)(((window && window < lane_rows ? window : lane_rows) + 63u) / 64u); }
// Splits of a layer's keys: a block per split where the window is short and lanes are few; up to 32 of them, and for more than four
// blocks in each as many as there are CTAs.  (Never more than 32: a step of one lane at 131072 keys took 1589 us, now 1025; at 32768 1023 and 899.)
int splits_of(int ctas, int m, int n_q, uint32_t window, uint32_t lane_rows) {
    const int most = ctas / (m * n_q / 8) - 1, blocks = blocks_of(window, lane_rows);
    int s = blocks <= 8 && m > 2 ? (blocks + 1) / 2 : blocks;
    if (s > FEW_SPLITS) s = blocks > FEW_SPLITS * FULL_SPLIT ? cdiv(blocks, FULL_SPLIT) : FEW_SPLITS;
    if (s > most) s = most;
    return s < 1 ? 1 : s;
}
// Whether the launches of run_layers take less time at full contexts, which is what the host knows of them.  A block of keys of a split takes
// 1.05 us from the fifth on, more than the attention launch needs for its share of them; a layer saves 7.5 us of hand-over for one and two lanes,
// 5.6 for three and 4.8 for four.  (One launch and launches, 35 layers of which 7 are full, tq2: two lanes x 131072 1189 and 1263 us; three x 65536
// 1187 and 1251, x 131072 1434 and 1345; four x 32768 1124 and 1209, x 65536 1284 and 1272, x 131072 1611 and 1406.)
bool launches_faster(int ctas, int m, int n_q, const LcStepLayer *layers, int n_layers) {
    const float saved = (m <= 2 ? 7.5f : (m == 3 ? 5.6f : 4.8f)) * (float)n_layers;
    int over = 0;
    for (int i = 0; i < n_layers; i++) {
        const int per = cdiv(blocks_of(layers[i].window, layers[i].lane_rows), splits_of(ctas, m, n_q, layers[i].window, layers[i].lane_rows));
        over += per > FULL_SPLIT ? per - FULL_SPLIT : 0;
    }
    return 1.05f * (float)over > saved;
}
size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

template <int BITS>
int launch_step(lc_kernels *k, lc_batch *b, LcStepParams &p) {
    using C = AttnCfg<HD, BITS>;
    using W = Wide<C>;
    const int ctas = k->ctx->sm_count, m = p.m, H = p.hidden;
    constexpr int STAGES = stages_of(BITS);
    auto up = [](int x) { return (x + 127) & ~127; };
    const int rb_h = H / 256 * 66, rb_o = (p.inter > p.n_q * HD ? p.inter : p.n_q * HD) / 256 * 66;
    const int ta = p.inter / 8 > (p.n_q + 2 * p.n_kv) * 16 ? p.inter / 8 : (p.n_q + 2 * p.n_kv) * 16;
    const int na = cdiv(ta, ctas);
    if (H / 16 > ctas || launches_faster(ctas, m, p.n_q, p.layer, p.n_layers)) return -1;
    int at = C::LUT_BYTES + C::Q_BYTES + HD * 4 + up(4 * H + na * 16 * rb_h);
    p.off_b = at;
    at += up(16 * rb_o);
    p.off_rot = at;
    at += m * 128 * 8;
    p.off_resid = at;
    at += up(m * H * 2);
    p.off_u = at;
    // work space: activations and sums of a projection, blocks of keys and their scratch, or the merge's groups
    if (na > MAX_TILES) return -1;
    const int units_b = (p.inter > p.n_q * HD ? p.inter : p.n_q * HD) / UNIT;
    const int red = (ST_NW + na) * RED_PART * 4, rows_a = m * (H * 2 + 64), rows_b = m * (units_b * UNIT * 2 + 64);
    p.off_red = up(rows_a > rows_b ? rows_a : rows_b);
    int work = p.off_red + red;
    for (int w : {STAGES * W::STAGE + W::SCRATCH + STAGES * 2 * W::KB * 4, (8 * PROW + ST_NT) * 4}) work = w > work ? w : work;
    const size_t smem = (size_t)at + up(work);
    if (smem + 3072 > k->ctx->smem_optin) return -1;
    size_t mail = 0;
    for (int i = 0; i < p.n_layers; i++) {
        LcStepLayer &L = p.layer[i];
        L.splits = (uint32_t)splits_of(ctas, m, p.n_q, L.window, L.lane_rows);
        L.mail = mail;
        mail += up256(mail_rows_bytes(m, H, p.inter, p.n_q, p.n_kv) + mail_partial_bytes(m, p.n_q, (int)L.splits));
    }
    auto kern = step_layers_kernel<BITS>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    LC_CUDA_TRY(cudaMemsetAsync(p.mail, 0xff, mail, b->stream));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(ST_NT + 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs run at once, or the launch fails
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LcPlain plain(b);   // (without the programmatic attribute it starts when its predecessor is complete)
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e == cudaErrorCooperativeLaunchTooLarge) {   // (part of the device only)
        cudaGetLastError();
        return -1;
    }
    LC_LAUNCH_CHECKED(e);
    b->dispatch_count++;
    return LC_OK;
}

}  // namespace

bool lc_step_small_supported(const lc_kernels *k, uint32_t hidden, uint32_t inter, uint32_t n_q, uint32_t n_kv, uint32_t head_dim,
                             uint32_t bits, uint32_t n_layers) {
    return head_dim == HD && lc_tq_attn_mma_supported(head_dim, bits) && n_kv >= 1 && n_q % (8 * n_kv) == 0 && hidden % 256 == 0 &&
           hidden <= (uint32_t)MAX_HIDDEN && inter % 256 == 0 && n_layers <= LC_STEP_MAX_LAYERS && k->kv_norm_mode == 0;
}

size_t lc_step_small_mail_bytes(const lc_kernels *k, uint32_t hidden, uint32_t inter, uint32_t n_q, uint32_t n_kv, uint32_t n_layers,
                                uint32_t max_lanes, const uint32_t *window, const uint32_t *lane_rows) {
    size_t most = 0;
    for (int m = 1; m <= (int)(max_lanes < LC_STEP_MAX_LANES ? max_lanes : LC_STEP_MAX_LANES); m++) {
        size_t n = 0;
        for (uint32_t i = 0; i < n_layers; i++)
            n += up256(mail_rows_bytes(m, (int)hidden, (int)inter, (int)n_q, (int)n_kv) +
                       mail_partial_bytes(m, (int)n_q, splits_of(k->ctx->sm_count, m, (int)n_q, window[i], lane_rows[i])));
        most = n > most ? n : most;
    }
    return most;
}

int lc_step_small_launch(lc_kernels *k, lc_batch *b, LcStepParams &p, uint32_t bits) {
    for (int i = 0; i < p.n_layers; i++) {
        const LcStepLayer &L = p.layer[i];
        for (const void *w : {(const void *)L.wq, (const void *)L.wk, (const void *)L.wv, (const void *)L.wo, (const void *)L.wgate, (const void *)L.wup,
                              (const void *)L.wdown, (const void *)L.attn_norm, (const void *)L.q_norm, (const void *)L.k_norm,
                              (const void *)L.post_attn_norm, (const void *)L.ffn_norm, (const void *)L.post_ffn_norm})
            if (!lc_aligned(w, 16)) return -1;
    }
    if (!lc_aligned(p.final_norm, 16) || !lc_aligned(p.embed, 2)) return -1;
    p.status = k->dev_status;
    p.wait_limit = k->test_wait_expiry ? 4096u : 1u << 21;
    p.never = k->test_wait_expiry ? 1u : 0u;
    switch (bits) {
        case 2: return launch_step<2>(k, b, p);
        case 3: return launch_step<3>(k, b, p);
        default: return launch_step<4>(k, b, p);
    }
}
