// Decode attention straight over TurboQuant codes, split-K across CTAs.
// Stands in for shaders/attention_flash_tq.metal:154-274 (flash_attention_tq)
// and :569-690 (flash_attention_tq_batched), plus the rotate -> attend ->
// inverse-rotate sequence the KV containers wrap around them
// (kv_cache/quant_cache.rs:565-596, kv_cache/quant_unified_pool.rs:218-256).
//
// Differences from the Metal design, all behaviour-preserving:
//  * one CTA serves every q-head that shares a kv-head, so a key/value row is
//    read from HBM once per group instead of once per q-head;
//  * the context is split across CTAs (grid.x) so one long sequence fills the
//    GPU; partial (max, sum, acc) triples are merged by a second kernel;
//  * in the fused form the query rotation runs in the prologue and the inverse
//    rotation + f16 store in the merge kernel, removing two launches and the
//    f32 round trips through rq / vacc.
#include <math.h>
#include <stdlib.h>

#include "lc_internal.h"
#include "attention_tq.h"
#include "split_merge.cuh"

namespace {

constexpr int NT = 256;
constexpr int NW = NT / 32;
constexpr int TILE = 32;  // keys per warp step: one key per lane in the QK phase


// In-place unnormalised FWHT on `rows` rows of HD floats in shared memory,
// cooperatively by the whole CTA.  Ends with a barrier.
template <int HD>
__device__ __forceinline__ void fwht_rows(float *sh, int rows) {
    const int pairs = rows * (HD / 2);
    for (int len = 1; len < HD; len <<= 1) {
        __syncthreads();
        for (int p = threadIdx.x; p < pairs; p += NT) {
            const int i = p & (len - 1);
            const int idx = ((p - i) << 1) + i;
            const float a = sh[idx], b = sh[idx + len];
            sh[idx] = a + b;
            sh[idx + len] = a - b;
        }
    }
    __syncthreads();
}

template <int HD, int BITS, int G>
__global__ void __launch_bounds__(NT) tq_attn_split_kernel(const TqAttnParams p) {
    lc_pdl_trigger();  // successors may be scheduled; they wait for this grid before reading its output
    lc_pdl_wait();     // everything below may read what the predecessor wrote
    constexpr int DPL = HD / 32;
    constexpr int CB = HD * BITS / 8;
    constexpr int NLEV = 1 << BITS;
    constexpr unsigned MASK = NLEV - 1;
    extern __shared__ __align__(16) float smem_f[];
    float *rq_s = smem_f;                   // [HD][G]
    float *lev_s = rq_s + HD * G;           // [16]
    float *pw_s = lev_s + 16;               // [NW][TILE][G]
    float *comb = pw_s + NW * TILE * G;     // [NW][G][HD] + m[NW][G] + l[NW][G]; also the rotation scratch

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t split = blockIdx.x;
    const uint32_t gchunks = (p.group + G - 1) / G;
    const uint32_t kv_head = blockIdx.y / gchunks, gchunk = blockIdx.y - kv_head * gchunks;
    const uint32_t lane_idx = blockIdx.z;
    const int gvalid = min((int)G, (int)(p.group - gchunk * G));
    const uint32_t qh0 = kv_head * p.group + gchunk * G;

    uint32_t pos, seq_len;
    if (p.positions) {
        pos = p.positions[lane_idx];
        seq_len = pos + 1u;
        if (p.ring == 0u && seq_len > p.lane_capacity) {   // never read past the lane's rows
            seq_len = p.lane_capacity;
            if (p.status && threadIdx.x == 0) atomicExch(p.status, LC_DEV_STATUS_POSITION);
        }
    } else {
        pos = p.current_pos + (p.row_positions ? lane_idx : 0u);
        seq_len = min(p.kv_len, pos + 1u);
    }
    const uint32_t win_start = (p.window > 0u && pos + 1u > p.window) ? (pos + 1u - p.window) : 0u;
    const uint32_t n_keys = seq_len > win_start ? seq_len - win_start : 0u;
    uint32_t per = (n_keys + p.n_splits - 1) / p.n_splits;
    per = (per + TILE - 1) & ~(uint32_t)(TILE - 1);
    const uint32_t k_begin = win_start + split * per;
    const uint32_t k_end = min(seq_len, k_begin + per);
    const size_t lane_base = (size_t)lane_idx * p.lane_capacity;

    // ---- prologue: query into shared memory as rq_s[d][g] (scaled) ----
    if (threadIdx.x < 16) lev_s[threadIdx.x] = threadIdx.x < NLEV ? p.levels[threadIdx.x] : 0.f;
    if (p.fused_q) {
        float *tmp = comb;  // [G][HD]
        for (int i = threadIdx.x; i < G * HD; i += NT) {
            const int g = i / HD, d = i - g * HD;
            float v = 0.f;
            if (g < gvalid) v = __half2float(p.q[((size_t)lane_idx * p.n_q + qh0 + g) * HD + d]) * p.signs[d];
            tmp[i] = v;
        }
        fwht_rows<HD>(tmp, G);
        const float f = p.scale / sqrtf((float)HD);
        for (int i = threadIdx.x; i < G * HD; i += NT) {
            const int g = i / HD, d = i - g * HD;
            rq_s[d * G + g] = tmp[i] * f;
        }
    } else {
        for (int i = threadIdx.x; i < G * HD; i += NT) {
            const int g = i / HD, d = i - g * HD;
            float v = 0.f;
            if (g < gvalid) v = p.rq[((size_t)lane_idx * p.n_q + qh0 + g) * HD + d] * p.scale;
            rq_s[d * G + g] = v;
        }
    }
    __syncthreads();

    float m_run[G], l_run[G], acc[G][DPL];
#pragma unroll
    for (int g = 0; g < G; g++) {
        m_run[g] = -INFINITY;
        l_run[g] = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; i++) acc[g][i] = 0.f;
    }
    float *pw = pw_s + warp * TILE * G;

    for (uint32_t t0 = k_begin + warp * TILE; t0 < k_end; t0 += NW * TILE) {
        // ---- QK: lane owns key t0 + lane, walks all HD codes ----
        const uint32_t t = t0 + lane;
        const bool valid = t < k_end;
        float s[G];
#pragma unroll
        for (int g = 0; g < G; g++) s[g] = 0.f;
        float vnorm = 0.f;
        if (valid) {
            const size_t slot = (lane_base + (p.ring ? t % p.ring : t)) * p.n_kv + kv_head;
            const uint32_t *kw = reinterpret_cast<const uint32_t *>(p.kc + slot * CB);
            constexpr int GW = (BITS == 3) ? 3 : 1;       // words per group
            constexpr int GC = GW * 32 / BITS;            // codes per group
#pragma unroll 2
            for (int grp = 0; grp < CB / 4 / GW; grp++) {
                uint32_t w[GW];
#pragma unroll
                for (int i = 0; i < GW; i++) w[i] = __ldg(kw + grp * GW + i);
#pragma unroll
                for (int c = 0; c < GC; c++) {
                    const int bo = c * BITS, wi = bo >> 5, sh = bo & 31;
                    unsigned code = w[wi] >> sh;
                    if (sh + BITS > 32) code |= w[wi + 1 < GW ? wi + 1 : wi] << (32 - sh);
                    code &= MASK;
                    const float lv = lev_s[code];
                    const float *rqd = rq_s + (grp * GC + c) * G;
#pragma unroll
                    for (int g = 0; g < G; g++) s[g] = fmaf(rqd[g], lv, s[g]);
                }
            }
            const float knorm = __half2float(p.kn[slot]);
            vnorm = __half2float(p.vn[slot]);
#pragma unroll
            for (int g = 0; g < G; g++) s[g] *= knorm;
        }
        // ---- online softmax for the tile ----
#pragma unroll
        for (int g = 0; g < G; g++) {
            float tm = valid ? s[g] : -INFINITY;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
            const float m_new = fmaxf(m_run[g], tm);  // finite: lane 0 of every tile is valid
            const float rescale = expf(m_run[g] - m_new);
            const float w = valid ? expf(s[g] - m_new) : 0.f;
            float ws = w;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
            l_run[g] = l_run[g] * rescale + ws;
            m_run[g] = m_new;
#pragma unroll
            for (int i = 0; i < DPL; i++) acc[g][i] *= rescale;
            pw[lane * G + g] = w * vnorm;
        }
        __syncwarp();
        // ---- PV: lane owns dims [lane*DPL, lane*DPL + DPL) ----
        const int nk = (int)min((uint32_t)TILE, k_end - t0);
        constexpr int BO = DPL * BITS;  // bits of codes owned by one lane
#pragma unroll 4
        for (int j = 0; j < nk; j++) {
            const uint32_t tj = t0 + j;
            const size_t slot = (lane_base + (p.ring ? tj % p.ring : tj)) * p.n_kv + kv_head;
            const uint8_t *vrow = p.vc + slot * CB;
            const unsigned bitoff = lane * BO, byte0 = bitoff >> 3, shb = bitoff & 7u;
            constexpr int NBYTES = (BO + 7 + 7) / 8 > 8 ? 8 : (BO + 7 + 7) / 8;
            unsigned long long bits = 0;
#pragma unroll
            for (int b = 0; b < NBYTES; b++)
                if (byte0 + b < (unsigned)CB) bits |= (unsigned long long)__ldg(vrow + byte0 + b) << (8 * b);
            bits >>= shb;
            float pj[G];
#pragma unroll
            for (int g = 0; g < G; g++) pj[g] = pw[j * G + g];
#pragma unroll
            for (int i = 0; i < DPL; i++) {
                const float lv = lev_s[(unsigned)(bits >> (i * BITS)) & MASK];
#pragma unroll
                for (int g = 0; g < G; g++) acc[g][i] = fmaf(pj[g], lv, acc[g][i]);
            }
        }
        __syncwarp();
    }

    // ---- merge the 8 warps of this CTA ----
    float *acc_s = comb;                       // [NW][G][HD]
    float *m_s = comb + NW * G * HD;           // [NW][G]
    float *l_s = m_s + NW * G;                 // [NW][G]
    __syncthreads();                           // comb may still hold the rotation scratch
#pragma unroll
    for (int g = 0; g < G; g++) {
        if (lane == 0) {
            m_s[warp * G + g] = m_run[g];
            l_s[warp * G + g] = l_run[g];
        }
#pragma unroll
        for (int i = 0; i < DPL; i++) acc_s[(warp * G + g) * HD + lane * DPL + i] = acc[g][i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < gvalid * HD; i += NT) {
        const int g = i / HD, d = i - g * HD;
        float gmax = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; w++) gmax = fmaxf(gmax, m_s[w * G + g]);
        float gsum = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float mw = m_s[w * G + g];
            const float f = (mw == -INFINITY) ? 0.f : expf(mw - gmax);
            gsum += f * l_s[w * G + g];
            o += f * acc_s[(w * G + g) * HD + d];
        }
        const size_t qh = (size_t)lane_idx * p.n_q + qh0 + g;
        if (p.direct_out) {
            p.out[qh * HD + d] = gsum > 0.f ? o / gsum : 0.f;
        } else {
            float *pp = p.partial + (qh * p.n_splits + split) * (size_t)(HD + 2);
            if (d == 0) {
                pp[0] = gmax;
                pp[1] = gsum;
            }
            pp[2 + d] = o;
        }
    }
}

// Merge n_splits partials of one (lane, q-head); optionally inverse-rotate and store f16 (fused form).
// grid = lanes * n_q.  The partials are added in groups of MERGE_RUN consecutive splits, then the groups in order (with at
// most MERGE_RUN splits that is plain split order, as the tensor-core kernel's own merge does it).  chunk != 0: the
// queue form's lanes differ in their number of partials.  Thread
// (column pair c, run r) adds run r, r + rows, ... of dims 2c, 2c + 1: the launch is a chain of L2 round trips, so all loads
// of a run are in flight together and the runs are spread over the block.
constexpr int MERGE_RUN = 8, MERGE_MAX_THREADS = 1024;
template <bool FUSED>
__global__ void __launch_bounds__(MERGE_MAX_THREADS)
tq_attn_merge_kernel(const float *__restrict__ partial, const float *__restrict__ signs, float *__restrict__ out_f32,
                     __half *__restrict__ out_f16, unsigned hd, unsigned n_splits, const uint32_t *__restrict__ positions,
                     unsigned n_q, unsigned lane_capacity, unsigned chunk) {
    lc_pdl_trigger();  // successors may be scheduled; they wait for this grid before reading its output
    lc_pdl_wait();     // everything below may read what the predecessor wrote
    __shared__ float sh[MERGE_MAX_THREADS];
    __shared__ float red[2 * MERGE_MAX_THREADS];        // [run row][hd]
    __shared__ float sum_s[MERGE_MAX_THREADS / 32];     // one per run row (hd >= 64: at most 32 rows)
    __shared__ float max_s[MERGE_MAX_THREADS / 32];
    const unsigned t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const size_t qh = blockIdx.x, row = hd + 2;
    const float *pp = partial + qh * n_splits * row;
    if (chunk) {   // queue form: only as many partials as the lane has items
        const unsigned keys = min(positions[qh / n_q] + 1u, lane_capacity);
        n_splits = lc_attn_items(keys, chunk);
    }
    const unsigned cols = hd / 2, c = t % cols, r0 = t / cols, rows = blockDim.x / cols;
    const unsigned runs = (n_splits + MERGE_RUN - 1) / MERGE_RUN;
    // first run's values are requested before anything else needs them
    float2 a[MERGE_RUN], ml[MERGE_RUN];
    auto load = [&](unsigned run) {
#pragma unroll
        for (int u = 0; u < MERGE_RUN; u++) {
            const unsigned s = run * MERGE_RUN + u;
            const bool ok = r0 < rows && s < n_splits;
            ml[u] = ok ? *reinterpret_cast<const float2 *>(pp + s * row) : make_float2(-INFINITY, 0.f);
            a[u] = ok ? *reinterpret_cast<const float2 *>(pp + s * row + 2 + 2 * c) : make_float2(0.f, 0.f);
        }
    };
    load(r0);
    float gmax = -INFINITY;
    for (unsigned s = t; s < n_splits; s += blockDim.x) gmax = fmaxf(gmax, pp[s * row]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    if (lane == 0) max_s[warp] = gmax;
    __syncthreads();
    for (unsigned w = 0; w < (blockDim.x + 31) / 32; w++) gmax = fmaxf(gmax, max_s[w]);
    float gsum = 0.f;
    float2 o = make_float2(0.f, 0.f);
    // Runs are added in order: each round of the block covers `rows` consecutive runs, whose sums meet in shared memory.
    for (unsigned run0 = 0; run0 < runs; run0 += rows) {
        if (run0) load(run0 + r0);
        float ps = 0.f;
        float2 po = make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < MERGE_RUN; u++) {
            const float f = (ml[u].x == -INFINITY) ? 0.f : expf(ml[u].x - gmax);
            ps += f * ml[u].y;
            po.x += f * a[u].x;
            po.y += f * a[u].y;
        }
        if (runs == 1) {
            gsum = ps;
            o = po;
            break;
        }
        if (r0 < rows) {
            if (c == 0) sum_s[r0] = ps;
            *reinterpret_cast<float2 *>(red + r0 * hd + 2 * c) = po;
        }
        __syncthreads();
        if (r0 == 0) {
            const unsigned n = runs - run0 < rows ? runs - run0 : rows;
            for (unsigned r = 0; r < n; r++) {
                const float2 v = *reinterpret_cast<const float2 *>(red + r * hd + 2 * c);
                gsum += sum_s[r];
                o.x += v.x;
                o.y += v.y;
            }
        }
        __syncthreads();
    }
    if (r0 == 0) {
        sh[2 * c] = gsum > 0.f ? o.x / gsum : 0.f;
        sh[2 * c + 1] = gsum > 0.f ? o.y / gsum : 0.f;
    }
    __syncthreads();
    const float v = t < hd ? sh[t] : 0.f;
    if (!FUSED) {
        if (t < hd) out_f32[qh * hd + t] = v;
        return;
    }
    // inverse rotation (threads past hd only take part in the barrier)
    const float w = lc_fwht_value(v, red, hd, t);
    if (t < hd) out_f16[qh * hd + t] = __float2half_rn(w * (1.0f / sqrtf((float)hd)) * signs[t]);
}

// The same sums, in the same order, with a warp per (lane, q-head): no barriers, and a run's loads in flight together.  The form
// for launches that have enough rows to fill the chip without splitting one; prefill of 256 rows
// x 8 heads over 4096 keys (9 splits, 19 MB of partials) 47.4 -> 39.3 us with it.  Dim 64 i + 2 lane + e is x[2 i + e].
constexpr unsigned MERGE_ROWS = 4, MERGE_ROWS_MAX_SPLITS = 32;
template <bool FUSED, int HD>
__global__ void __launch_bounds__(MERGE_ROWS * 32)
tq_attn_merge_rows_kernel(const float *__restrict__ partial, const float *__restrict__ signs, float *__restrict__ out_f32,
                          __half *__restrict__ out_f16, unsigned rows, unsigned n_splits, const uint32_t *__restrict__ positions,
                          unsigned n_q, unsigned lane_capacity, unsigned chunk) {
    constexpr int P = HD / 64, BATCH = HD > 256 ? 4 : 8;   // float2 per lane; splits loaded together
    lc_pdl_trigger();
    const unsigned lane = threadIdx.x & 31, qh = blockIdx.x * MERGE_ROWS + (threadIdx.x >> 5);
    if (qh >= rows) return;
    lc_pdl_wait();
    constexpr size_t row = HD + 2;
    const float *pp = partial + (size_t)qh * n_splits * row;
    if (chunk) n_splits = lc_attn_items(min(positions[qh / n_q] + 1u, lane_capacity), chunk);
    const float2 ml = lane < n_splits ? *reinterpret_cast<const float2 *>(pp + lane * row) : make_float2(-INFINITY, 0.f);
    // Small heads leave registers for a second batch on its way while the first is added (200 rows of 8 heads at head_dim 128 over 2000
    // keys 21.1 -> 20.0 us; at 256 it leaves an SM fewer warps, 29.3 -> 30.8).
    constexpr int NBUF = HD <= 128 ? 2 : 1;
    float2 a[NBUF][BATCH][P];
    auto load = [&](float2 (&v)[BATCH][P], unsigned s0) {
#pragma unroll
        for (int u = 0; u < BATCH; u++)
#pragma unroll
            for (int i = 0; i < P; i++)
                v[u][i] = s0 + u < n_splits ? *reinterpret_cast<const float2 *>(pp + (s0 + u) * row + 2 + 64 * i + 2 * lane) : make_float2(0.f, 0.f);
    };
    load(a[0], 0);
    if (NBUF == 2 && BATCH < n_splits) load(a[NBUF - 1], BATCH);
    float gmax = ml.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    const float fl = (ml.x == -INFINITY) ? 0.f : expf(ml.x - gmax);
    float gsum = 0.f, ps = 0.f, x[2 * P], po[2 * P];
#pragma unroll
    for (int i = 0; i < 2 * P; i++) x[i] = po[i] = 0.f;
    auto add = [&](const float2 (&v)[BATCH][P], unsigned s0) {
#pragma unroll
        for (int u = 0; u < BATCH; u++) {
            const float f = __shfl_sync(0xffffffffu, fl, (s0 + u) & 31), l = __shfl_sync(0xffffffffu, ml.y, (s0 + u) & 31);
            if (s0 + u < n_splits) {
                ps += f * l;
#pragma unroll
                for (int i = 0; i < P; i++) {
                    po[2 * i] += f * v[u][i].x;
                    po[2 * i + 1] += f * v[u][i].y;
                }
            }
        }
        if ((s0 + BATCH) % MERGE_RUN == 0 || s0 + BATCH >= n_splits) {   // a run is complete
            gsum += ps;
            ps = 0.f;
#pragma unroll
            for (int i = 0; i < 2 * P; i++) {
                x[i] += po[i];
                po[i] = 0.f;
            }
        }
    };
    for (unsigned s0 = 0; s0 < n_splits; s0 += NBUF * BATCH) {
#pragma unroll
        for (int n = 0; n < NBUF; n++) {
            const unsigned s = s0 + n * BATCH;
            if (s >= n_splits) break;
            add(a[n], s);
            if (s + NBUF * BATCH < n_splits) load(a[n], s + NBUF * BATCH);
        }
    }
#pragma unroll
    for (int i = 0; i < 2 * P; i++) x[i] = gsum > 0.f ? x[i] / gsum : 0.f;
    if (!FUSED) {
#pragma unroll
        for (int i = 0; i < P; i++) *reinterpret_cast<float2 *>(out_f32 + (size_t)qh * HD + 64 * i + 2 * lane) = make_float2(x[2 * i], x[2 * i + 1]);
        return;
    }
    // inverse rotation: butterflies in ascending stride
#pragma unroll
    for (int i = 0; i < P; i++) {
        const float u = x[2 * i], v = x[2 * i + 1];
        x[2 * i] = __fadd_rn(u, v);
        x[2 * i + 1] = __fsub_rn(u, v);
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const bool upper = lane & m;
#pragma unroll
        for (int i = 0; i < 2 * P; i++) {
            const float o = __shfl_xor_sync(0xffffffffu, x[i], m);
            x[i] = upper ? __fsub_rn(o, x[i]) : __fadd_rn(x[i], o);
        }
    }
    if constexpr (P > 1) {
#pragma unroll
        for (int len = 2; len < 2 * P; len <<= 1)
#pragma unroll
            for (int i = 0; i < 2 * P; i++)
                if (!(i & len)) {
                    const float u = x[i], v = x[i + len];
                    x[i] = __fadd_rn(u, v);
                    x[i + len] = __fsub_rn(u, v);
                }
    }
    const float inv = 1.0f / sqrtf((float)HD);
#pragma unroll
    for (int i = 0; i < P; i++) {
        const float2 sg = *reinterpret_cast<const float2 *>(signs + 64 * i + 2 * lane);
        *reinterpret_cast<__half2 *>(out_f16 + (size_t)qh * HD + 64 * i + 2 * lane) = __floats2half2_rn(x[2 * i] * inv * sg.x, x[2 * i + 1] * inv * sg.y);
    }
}

// Many splits of few heads (split_merge.cuh).  One lane of 32768 keys, 148 splits of 8 heads: 18.8 -> 13.0 us with the launch before it; inverse
// rotation by shuffles and one barrier in place of a barrier per stage: 12.36 -> 12.25, tq4 at head_dim 128 10.9 -> 10.7.
template <bool FUSED>
__global__ void __launch_bounds__(MC_THREADS)
tq_attn_merge_cluster_kernel(const float *__restrict__ partial, const float *__restrict__ signs, float *__restrict__ out_f32,
                             __half *__restrict__ out_f16, unsigned hd, unsigned n_splits) {
    lc_pdl_trigger();
    __shared__ ClusterMerge sh;
    const size_t qh = blockIdx.x / MC, row = hd + 2;
    const float *pp = partial + qh * n_splits * row;
    float2 o = make_float2(0.f, 0.f);
    float gsum = 0.f;
    const unsigned t = threadIdx.x;
    const bool mine = cluster_merge(
        sh, hd, n_splits, [&](unsigned s) { return *reinterpret_cast<const float2 *>(pp + s * row); },
        [&](unsigned s, unsigned c) { return *reinterpret_cast<const float2 *>(pp + s * row + 2 + 2 * c); }, o, gsum);
    if (blockIdx.x % MC != 0) return;
    if (mine) {
        o.x = gsum > 0.f ? o.x / gsum : 0.f;
        o.y = gsum > 0.f ? o.y / gsum : 0.f;
        if (!FUSED) *reinterpret_cast<float2 *>(out_f32 + qh * hd + 2 * t) = o;
        else *reinterpret_cast<float2 *>(sh.fwht + 2 * t) = o;
    }
    if (!FUSED) return;
    __syncthreads();
    if (hd <= MC_THREADS) {   // inverse rotation, a dim per thread (threads past hd only take part in the barrier)
        const float w = lc_fwht_value(t < hd ? sh.fwht[t] : 0.f, sh.red, hd, t);
        if (t < hd) out_f16[qh * hd + t] = __float2half_rn(w * (1.0f / sqrtf((float)hd)) * signs[t]);
        return;
    }
    // a stage after the other; a thread has at most one pair
    for (unsigned len = 1; len < hd; len <<= 1) {
        if (t < hd / 2) {
            const unsigned i = (t & ~(len - 1)) * 2 + (t & (len - 1));
            const float x = sh.fwht[i], y = sh.fwht[i + len];
            sh.fwht[i] = __fadd_rn(x, y);
            sh.fwht[i + len] = __fsub_rn(x, y);
        }
        __syncthreads();
    }
    for (unsigned d = t; d < hd; d += MC_THREADS) out_f16[qh * hd + d] = __float2half_rn(sh.fwht[d] * (1.0f / sqrtf((float)hd)) * signs[d]);
}

// block of the merge launch: one run of splits per hd / 2 threads, at least hd threads
unsigned merge_threads(unsigned hd, unsigned n_splits) {
    const unsigned runs = (n_splits + MERGE_RUN - 1) / MERGE_RUN;
    unsigned t = hd / 2 * runs;
    if (t < hd) t = hd;
    return t > MERGE_MAX_THREADS ? MERGE_MAX_THREADS : t;
}

template <bool FUSED>
int launch_merge_rows(lc_batch *b, const float *partial, const float *signs, void *out, unsigned hd, unsigned rows, unsigned n_splits,
                      const uint32_t *positions, unsigned n_q, unsigned lane_capacity, unsigned chunk) {
    auto go = [&](auto kern) -> int {
        LC_LAUNCH_CHECKED(lc_launch(kern, dim3((rows + MERGE_ROWS - 1) / MERGE_ROWS), dim3(MERGE_ROWS * 32), 0, b, partial, signs, (float *)(FUSED ? nullptr : out),
                                    (__half *)(FUSED ? out : nullptr), rows, n_splits, positions, n_q, lane_capacity, chunk));
        return LC_OK;
    };
    switch (hd) {
        case 64: return go(tq_attn_merge_rows_kernel<FUSED, 64>);
        case 128: return go(tq_attn_merge_rows_kernel<FUSED, 128>);
        case 256: return go(tq_attn_merge_rows_kernel<FUSED, 256>);
        default: return go(tq_attn_merge_rows_kernel<FUSED, 512>);
    }
}

// A warp per row while that gives every SM a block; with fewer rows a block each is the shorter chain.
int launch_merge(lc_batch *b, bool fused, const float *partial, const float *signs, void *out, unsigned hd, unsigned rows, unsigned n_splits,
                 const uint32_t *positions, unsigned n_q, unsigned lane_capacity, unsigned chunk, unsigned sms) {
    if (n_splits <= MERGE_ROWS_MAX_SPLITS && rows >= MERGE_ROWS * sms / 2 && lc_aligned(out, 8) && (!fused || lc_aligned(signs, 8))) {
        return fused ? launch_merge_rows<true>(b, partial, signs, out, hd, rows, n_splits, positions, n_q, lane_capacity, chunk)
                     : launch_merge_rows<false>(b, partial, signs, out, hd, rows, n_splits, positions, n_q, lane_capacity, chunk);
    }
    if (chunk == 0 && cluster_merge_fits(b->ctx, rows, n_splits, hd) && lc_aligned(out, 8)) {
        if (fused)
            LC_LAUNCH_CHECKED(launch_cluster_merge(tq_attn_merge_cluster_kernel<true>, rows, b, partial, signs, nullptr, (__half *)out, hd, n_splits));
        else
            LC_LAUNCH_CHECKED(launch_cluster_merge(tq_attn_merge_cluster_kernel<false>, rows, b, partial, nullptr, (float *)out, nullptr, hd, n_splits));
        return LC_OK;
    }
    if (fused)
        LC_LAUNCH_CHECKED(lc_launch(tq_attn_merge_kernel<true>, dim3(rows), dim3(merge_threads(hd, n_splits)), 0, b, partial, signs, nullptr, (__half *)out, hd, n_splits, positions, n_q, lane_capacity, chunk));
    else
        LC_LAUNCH_CHECKED(lc_launch(tq_attn_merge_kernel<false>, dim3(rows), dim3(merge_threads(hd, n_splits)), 0, b, partial, nullptr, (float *)out, nullptr, hd, n_splits, positions, n_q, lane_capacity, chunk));
    return LC_OK;
}

template <int HD, int BITS, int G>
int launch_split(lc_batch *b, const TqAttnParams &p, dim3 grid) {
    const size_t comb = (size_t)NW * G * HD + 2 * NW * G;
    const size_t floats = (size_t)HD * G + 16 + (size_t)NW * TILE * G + comb;
    const size_t smem = floats * sizeof(float);
    auto kern = tq_attn_split_kernel<HD, BITS, G>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    LC_LAUNCH_CHECKED(lc_launch(kern, dim3(grid), dim3(NT), smem, b, p));
    LC_CHECK_LAUNCH("flash_attention_tq");
    b->dispatch_count++;
    return LC_OK;
}

template <int HD, int BITS>
int launch_split_g(lc_batch *b, const TqAttnParams &p, dim3 grid, int g) {
    switch (g) {
        case 1: return launch_split<HD, BITS, 1>(b, p, grid);
        case 2: return launch_split<HD, BITS, 2>(b, p, grid);
        case 4: return launch_split<HD, BITS, 4>(b, p, grid);
        default: return launch_split<HD, BITS, 8>(b, p, grid);
    }
}

template <int HD>
int launch_split_b(lc_batch *b, const TqAttnParams &p, dim3 grid, int g, unsigned bits) {
    switch (bits) {
        case 2: return launch_split_g<HD, 2>(b, p, grid, g);
        case 3: return launch_split_g<HD, 3>(b, p, grid, g);
        default: return launch_split_g<HD, 4>(b, p, grid, g);
    }
}

// What the tensor-core kernels take, for the choice between their forms, in ns (keys: ps).  Fitted to graphs of calls on one B200, 8 heads on one kv head,
// after the kernels' last change: decode kernel 1 .. 128 lanes x 256 .. 8192 keys at every split count, prefill kernel 8 .. 256 rows x 300 ..
// 8192 keys at 1 .. 32 splits; both within 3 % in the mean.
struct AttnTimes {
    uint32_t start, wave, key;            // decode kernel: a launch, each further wave, a key of a CTA
    uint32_t pf_start, pf_wave, pf_tile;  // prefill kernel: the same, a tile of keys
};
constexpr uint32_t ATTN_CLUSTER = 500;   // splits merged by the launch itself
uint32_t attn_merge_ns(const lc_ctx *ctx, uint32_t rows, uint32_t splits, uint32_t hd) {   // splits merged by another launch
    return cluster_merge_fits(ctx, rows, splits, hd) ? 2700 : 850 + 94 * splits;
}
AttnTimes attn_times(uint32_t hd, uint32_t bits) {
    if (hd == 512) return {8800, 9200, bits == 2 ? 32400u : 35000u, 0, 0, 0};   // (the prefill kernel has no such heads)
    if (hd == 256) {
        if (bits == 2) return {7000, 7500, 7900, 14300, 9000, 1320};
        return {7000, 7500, bits == 3 ? 16600u : 15300u, 13600, 7700, 1500};
    }
    return {5600, 5500, bits == 2 ? 8900u : bits == 3 ? 10800u : 9300u, 11200, 6300, 1490};
}

// Common host path.  `q_f16`/`out_f16` select the fused form.
int tq_attention(const char *name, lc_kernels *k, lc_batch *b, const lc_buf *rq_or_q, bool fused,
                 const lc_buf *kc, const lc_buf *kn, const lc_buf *vc, const lc_buf *vn, const lc_buf *levels,
                 const lc_buf *signs, lc_buf *out, const lc_buf *positions, uint32_t hd, uint32_t kv_len,
                 uint32_t current_pos, uint32_t lane_capacity, uint32_t n_q, uint32_t n_kv, uint32_t window,
                 uint32_t bits, uint32_t n_lanes, uint32_t ring, float scale, uint32_t n_rows = 0,
                 const lc_buf *qfrag = nullptr) {
    // n_rows != 0: prefill / multi-row verify over one cache: row r at position current_pos + r (n_lanes is ignored)
    const bool prefill = n_rows != 0;
    if (prefill) n_lanes = n_rows;
    if (!k || !b || !rq_or_q || !kc || !kn || !vc || !vn || !levels || !out || (fused && !signs))
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: NULL argument", name);
    if (bits < 2 || bits > 4) return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: bits %u not in 2..=4", name, bits);
    if (hd != 64 && hd != 128 && hd != 256 && hd != 512)
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: head_dim %u must be 64, 128, 256 or 512", name, hd);
    LC_REQUIRE(n_kv >= 1 && n_q >= 1 && n_q % n_kv == 0, "%s: num_q_heads %u must be a multiple of num_kv_heads %u",
               name, n_q, n_kv);
    if (n_lanes == 0) return LC_OK;
    const size_t cb = (size_t)hd * bits / 8;
    const size_t qn = (size_t)n_lanes * n_q * hd;
    LC_REQUIRE(rq_or_q->bytes >= qn * (fused ? 2 : 4) && out->bytes >= qn * (fused ? 2 : 4),
               "%s: query/output buffers too small", name);
    LC_REQUIRE(levels->bytes >= (4u << bits), "%s: levels buffer too small", name);
    if (fused) LC_REQUIRE(signs->bytes >= hd * 4u, "%s: signs buffer too small", name);
    // Rows a launch may touch: single form reads slots < min(kv_len, pos+1) (or < ring).
    size_t rows;
    uint32_t len_max, seq_max = 0;   // the most keys a row attends; one cache: the keys in it
    if (positions) {
        LC_REQUIRE(positions->bytes >= (size_t)n_lanes * 4, "%s: positions buffer too small", name);
        LC_REQUIRE(ring <= lane_capacity, "%s: ring %u exceeds lane capacity %u", name, ring, lane_capacity);
        rows = (size_t)n_lanes * lane_capacity;
        len_max = ring ? ring : lane_capacity;
    } else {
        const uint32_t last_pos = current_pos + (prefill ? n_rows - 1 : 0);   // the row that sees the most keys
        const uint32_t seq_len = kv_len < last_pos + 1 ? kv_len : last_pos + 1;
        seq_max = seq_len;
        rows = ring ? (ring < seq_len ? ring : seq_len) : seq_len;
        const uint32_t ws = (window > 0 && last_pos + 1 > window) ? last_pos + 1 - window : 0;
        len_max = seq_len > ws ? seq_len - ws : 0;
        lane_capacity = 0;
    }
    if (window > 0 && len_max > window) len_max = window;
    LC_REQUIRE(kc->bytes >= rows * n_kv * cb && vc->bytes >= rows * n_kv * cb && kn->bytes >= rows * n_kv * 2 &&
                   vn->bytes >= rows * n_kv * 2,
               "%s: KV buffers hold fewer than %zu rows", name, rows);
    LC_REQUIRE(lc_aligned(kc->dptr, 16) && lc_aligned(vc->dptr, 16), "%s: code buffers must be 16-byte aligned", name);
    LC_REQUIRE(lc_aligned(rq_or_q->dptr, fused ? 2 : 4) && lc_aligned(out->dptr, fused ? 2 : 4) &&
                   lc_aligned(levels->dptr, 4) && (!fused || lc_aligned(signs->dptr, 4)) && lc_aligned(kn->dptr, 2) &&
                   lc_aligned(vn->dptr, 2),
               "%s: a buffer is not aligned to its element size", name);

    const uint32_t group = n_q / n_kv;
    int g = group >= 8 ? 8 : (group > 4 ? 8 : (group > 2 ? 4 : (group > 1 ? 2 : 1)));
    // Head sizes 128 / 256 / 512 run on the tensor-core kernel (8 heads per CTA; a group of fewer heads leaves MMA columns
    // empty, and a single head per kv-head is left to the CUDA cores).  It loads queries and signs as 16-byte vectors and
    // 32-key tiles that wrap at most once: other buffers and rings take the CUDA-core kernel, as does LOCAL_CUDA_ATTN_MMA=0.
    static const bool mma_allowed = []() { const char *e = getenv("LOCAL_CUDA_ATTN_MMA"); return !(e && e[0] == '0'); }();
    const bool use_mma = mma_allowed && lc_tq_attn_mma_supported(hd, bits) && group >= 2 && (ring == 0 || ring >= 32) &&
                         lc_aligned(rq_or_q->dptr, 16) && (!fused || lc_aligned(signs->dptr, 16));
    if (use_mma) g = 8;
    const uint32_t gchunks = (group + g - 1) / g;
    const uint32_t base = n_lanes * n_kv * gchunks;
    const uint32_t sms = (uint32_t)k->ctx->sm_count;
    uint32_t want = (2u * sms + base - 1) / base;
    uint32_t by_len = (len_max + NW * TILE - 1) / (NW * TILE);
    if (by_len < 1) by_len = 1;
    uint32_t n_splits = want < by_len ? want : by_len;
    if (n_splits < 1) n_splits = 1;
    if (n_splits > 64) n_splits = 64;
    uint32_t chunk = 0;
    // The tensor-core kernel merges up to 8 splits itself (one thread-block cluster per lane and kv head, exchange
    // through distributed shared memory, inverse rotation in the kernel): one launch instead of split + merge, the same
    // arithmetic in the same order, bit-identical output.  LOCAL_CUDA_ATTN_CLUSTER=0 selects the two-launch form.
    static const bool cluster_allowed = []() { const char *e = getenv("LOCAL_CUDA_ATTN_CLUSTER"); return !(e && e[0] == '0'); }();
    const bool clusters = use_mma && cluster_allowed && lc_aligned(out->dptr, 16) && (!fused || lc_aligned(signs->dptr, 16));
    uint64_t grid_cost = ~0ull;
    // (Pools of tq2 rows at head_dim 256 are counted in keys of 8.5 ns, an older fit that chooses as well there: over 24 pools 0.5 % above the faster form in
    // the mean, 0.6 with the times above.)
    const bool counted = positions && bits == 2 && hd == 256;
    const AttnTimes t = counted ? AttnTimes{700, 1050, 1000, 0, 0, 0} : attn_times(hd, bits);
    const uint32_t cluster_cost = counted ? 0 : ATTN_CLUSTER;
    auto keys_ns = [&](uint64_t keys) -> uint64_t { return keys * t.key / 1000u; };
    if (use_mma) {
        // One CTA per SM (shared memory), so the launch runs in whole waves.  Pick the split count that minimises their time.
        // Short contexts split down to two 32-key tiles per CTA (two warps that have the table's banks to themselves finish a
        // tile sooner than eight), but into no more splits than one launch merges; long ones to half the warps.
        uint32_t max_s = len_max < 4096 ? len_max / 64u : len_max / 128u;
        if (len_max < 4096 && max_s > 8) max_s = 8;
        if (max_s < 1) max_s = 1;
        if (max_s > sms) max_s = sms;
        // The lanes of a pool are as a rule shorter than its rows: splits save less there, and a merge costs the same (4 lanes of 16 heads over 7605 rows, full and
        // ragged together: 8 splits in one launch 25.2 us, 18 and a merge 26.5).
        auto merge_ns = [&](uint32_t s) -> uint32_t { return counted ? 640u : attn_merge_ns(b->ctx, (uint32_t)(qn / hd), s, hd) + (positions ? 2500u : 0u); };
        // Up to 8 splits are a cluster, and of those fewer fit at once (17 lanes x 512 keys: 8 splits 17.2 us, 6 splits 9.3).
        for (uint32_t s = 1; s <= max_s; s++) {
            const bool one_launch = s <= 8 && clusters;
            const uint64_t waves = one_launch ? (base + k->cluster_cap[s] - 1) / k->cluster_cap[s] : ((uint64_t)base * s + sms - 1) / sms;
            const uint64_t cost = t.start + waves * keys_ns((len_max + s - 1) / s) + (waves - 1) * t.wave + (s == 1 ? 0u : one_launch ? cluster_cost : merge_ns(s));
            if (cost < grid_cost) { grid_cost = cost; n_splits = s; }
        }
    }
    // The two forms below need room for partials where the splits above may need none, and scratch memory cannot grow while a graph
    // is recorded: a call that was not made outside capture first keeps the splits.
    auto partials_fit = [&](uint32_t splits, size_t counters) {
        return !b->capturing || (qn / hd * splits * (size_t)(hd + 2) * sizeof(float) <= k->scratch_bytes && counters <= k->counters_len);
    };
    // Queue form for pools of lanes that attend all of their keys.  Lanes differ in length, which the host cannot see, and
    // equal splits per lane leave most SMs waiting for the longest lane; so one persistent CTA per SM draws items of at
    // most `chunk` keys; a merge launch follows.  The chunk minimises the sum of two estimates: every lane full, and lane lengths spread evenly up to
    // the longest.  The splits above take their longest lane's time in both, in one launch, and stay unless the queue promises less: measured full / ragged,
    // 32 lanes x 8192 tq2 keys 25.7 / 21.0 us against 34.7 / 21.8 for the queue, 64 lanes 40.1 / 38.3 against 50.7 / 29.4,
    // 64 lanes of tq4 keys 70.9 / 68.4 against 80.4 / 44.0; over 76 pools the choice takes 0.7 % longer than the faster form
    // and cut in the mean, 8 % at most.  (In a pool of few lanes the longest is often short, too, and the splits then gain as much: 17 lanes x 7600 tq4 keys at
    // head_dim 128, two kv heads, 30.5 / 17.7 as splits, 35.9 / 20.7 as items; but 18 lanes x 7010 at head_dim 512 104.5 together, 95.9.)
    if (use_mma && positions && window == 0 && ring == 0 && n_lanes <= LC_ATTN_QUEUE_LANES && base * 16u >= sms && len_max > 2048) {
        // an item after a CTA's first costs about three quarters of a launch's start more
        const uint32_t lo_s = len_max > 32u * 2048u ? 32u : (len_max + 4095) / 4096, item = counted ? 620u : t.start * 3u / 4u,
                       launches = counted ? 700u + 640u : t.start + 3500u + 6u * hd, enough = counted ? 100u : 99u;
        uint64_t best_cost = ~0ull / 128u;
        uint32_t best_chunk = 0;
        for (uint32_t s = lo_s; s <= 32; s++) {
            uint32_t per = ((len_max - 64u) / s + 255u) & ~255u;   // whole rounds of eight warps x 32 keys
            if (per < 256u) per = 256u;
            const uint64_t rounds = ((uint64_t)base * s + sms - 1) / sms, one = keys_ns(per), full = rounds * one + (rounds - 1) * item;
            const uint64_t mean = base * (keys_ns(len_max) + (uint64_t)item * (s + 1)) / 2 / sms;
            const uint64_t cost = full + (mean > one ? mean : one) + 2u * launches;
            if (cost * 100u < best_cost * enough) { best_cost = cost; best_chunk = per + 64u; }   // (a few keys over do not make another item; of near equals the fewer items)
        }
        const uint32_t most = best_chunk ? (len_max + best_chunk - 1) / best_chunk : 1u;
        if (best_cost < 2u * grid_cost && partials_fit(most, (size_t)n_kv * gchunks)) {
            chunk = best_chunk;
            n_splits = most;
        }
    }
    // Chunks of several rows: the prefill kernel shares each decoded key among 128 MMA rows, but takes longer before and after its key tiles and
    // leaves a merge launch.  Fewer than half a tile of rows, and chunks whose rows the decode kernel's
    // CTAs finish sooner, stay there (tq2): 64 rows over 400 keys 9.7 us against 15.9, 256 over 300 19.0 against 18.1, 256 over
    // 4096 77 against 30; tq4 128 over 2000 39 against 26, at head_dim 128 64 over 8192 46 against 21.  Over 360 chunks the choice takes 0.7 % longer than
    // the faster kernel at its best split in the mean, 19 % at most (16 tq3 rows over 8192 at head_dim 128: 22.0 against 18.5).
    uint32_t pf_heads = 1, pf_tiles = 0;
    if (prefill && use_mma && lc_tq_attn_prefill_supported(hd, bits)) {
        const uint32_t heads = group < 8 ? group : 8;
        while (pf_heads < heads) pf_heads <<= 1;
        const uint32_t rows_per_tile = 128 / pf_heads;
        if (n_rows * 2 >= rows_per_tile) {
            pf_tiles = (n_rows + rows_per_tile - 1) / rows_per_tile;
            const uint32_t ctas = n_kv * gchunks * pf_tiles, tile = lc_tq_attn_prefill_tile_keys(hd, bits);
            uint32_t seen = len_max + (rows_per_tile < n_rows ? rows_per_tile : n_rows);   // keys of a tile of rows, at most
            if (seen > seq_max) seen = seq_max;
            const uint32_t key_tiles = (seen + tile - 1) / tile;
            uint32_t most = ctas < sms ? sms / ctas : 1;   // one wave
            if (most > key_tiles) most = key_tiles;
            if (most > MERGE_ROWS_MAX_SPLITS) most = MERGE_ROWS_MAX_SPLITS;
            // The merge launch's blocks (MERGE_ROWS rows each) become resident ahead of their turn on the SMs that this launch leaves free, up to five on one, and
            // read all their partials through those: some 90 bytes a ns and SM (64 rows of 8 heads over 4096 keys: 24 splits on 96 SMs 21.5 us, 32 on 128 26.0).
            const uint32_t merge_blocks = (n_rows * n_q + MERGE_ROWS - 1) / MERGE_ROWS, split_bytes = hd * 4u;
            const uint64_t waves = (ctas + sms - 1) / sms;
            uint64_t best = ~0ull / 128u;
            uint32_t splits = 1;
            for (uint32_t sp = most; sp >= 1; sp--) {   // (of near equals the most splits: the first rows of a chunk see fewer keys)
                const uint32_t free = (uint32_t)waves * sms - ctas * sp;
                uint32_t crowd = 0;
                if (free) crowd = merge_blocks > 5u * free ? 5u : (merge_blocks + free - 1) / free;
                const uint64_t cost = t.pf_start + (waves - 1) * t.pf_wave + waves * ((key_tiles + sp - 1) / sp) * t.pf_tile +
                                      (uint64_t)n_rows * n_q * sp * split_bytes * 11u / 100000u + crowd * MERGE_ROWS * 4u * sp * hd / 90u;
                if (cost * 102u < best * 100u) { best = cost; splits = sp; }
            }
            if (best < grid_cost && partials_fit(splits, 0))
                n_splits = splits;
            else
                pf_tiles = 0;
        }
    }
    const bool pf = pf_tiles != 0;
    const bool queue = chunk != 0;
    const bool direct = !queue && !pf && n_splits == 1 && !fused;
    const bool cluster_merge = clusters && !queue && !pf && n_splits <= 8;

    if (!direct && !cluster_merge) {
        const size_t rows_y = (size_t)n_kv * gchunks;
        int st = lc_reserve_scratch(k, b, qn / hd * n_splits * (size_t)(hd + 2) * sizeof(float), queue ? rows_y : 0);
        if (st != LC_OK) return st;
    }
    TqAttnParams p;
    p.rq = fused ? nullptr : (const float *)rq_or_q->dptr;
    p.q = fused ? (const __half *)rq_or_q->dptr : nullptr;
    p.signs = signs ? (const float *)signs->dptr : nullptr;
    p.kc = (const uint8_t *)kc->dptr;
    p.vc = (const uint8_t *)vc->dptr;
    p.kn = (const __half *)kn->dptr;
    p.vn = (const __half *)vn->dptr;
    p.levels = (const float *)levels->dptr;
    p.out = (direct || (cluster_merge && !fused)) ? (float *)out->dptr : nullptr;
    p.out_f16 = (cluster_merge && fused) ? (__half *)out->dptr : nullptr;
    p.queue_chunk = chunk;
    p.n_lanes = n_lanes;
    p.counters = k->counters;
    p.pf_heads = pf_heads;
    p.wait_limit = k->test_wait_expiry ? 4096u : 1u << 22;
    p.extra_arrivals = k->test_wait_expiry ? 1u : 0u;
    p.cluster_merge = cluster_merge ? 1 : 0;
    p.partial = (float *)k->scratch;
    p.positions = positions ? (const uint32_t *)positions->dptr : nullptr;
    p.kv_len = kv_len;
    p.current_pos = current_pos;
    p.row_positions = prefill ? 1 : 0;
    p.lane_capacity = lane_capacity;
    p.n_q = n_q;
    p.n_kv = n_kv;
    p.window = window;
    p.ring = ring;
    p.n_splits = n_splits;
    p.group = group;
    p.fused_q = fused ? 1 : 0;
    p.direct_out = direct ? 1 : 0;
    p.scale = scale;
    p.status = k->dev_status;
    p.qfrag = nullptr;
    p.early_kv = (qfrag && use_mma && positions) ? 1u : 0u;   // only the decode step passes fragments: its positions are a step input
    if (qfrag && use_mma && fused && lc_qfrag_supported(hd, bits, n_q, n_kv)) {
        LC_REQUIRE(qfrag->bytes >= qn * 4, "%s: query fragment buffer too small", name);
        p.qfrag = (const uint4 *)qfrag->dptr;
    }
    dim3 grid(n_splits, n_kv * gchunks, n_lanes);
    if (queue) {
        const uint32_t per_y = sms / grid.y ? sms / grid.y : 1u;
        grid = dim3(per_y < n_lanes * n_splits ? per_y : n_lanes * n_splits, grid.y, 1);
    }
    int st;
    if (pf) {
        st = lc_tq_attn_prefill_launch(b, p, dim3(n_splits, n_kv * gchunks, pf_tiles), hd, bits);
    } else if (use_mma) {
        st = lc_tq_attn_mma_launch(b, p, grid, hd, bits);
    } else {
        switch (hd) {
            case 64: st = launch_split_b<64>(b, p, grid, g, bits); break;
            case 128: st = launch_split_b<128>(b, p, grid, g, bits); break;
            case 256: st = launch_split_b<256>(b, p, grid, g, bits); break;
            default: st = launch_split_b<512>(b, p, grid, g, bits); break;
        }
    }
    if (st != LC_OK || direct || cluster_merge) return st;
    st = launch_merge(b, fused, (const float *)k->scratch, fused ? (const float *)signs->dptr : nullptr, out->dptr, hd, n_lanes * n_q, n_splits, p.positions,
                      n_q, lane_capacity, chunk, sms);
    if (st != LC_OK) return st;
    LC_CHECK_LAUNCH("flash_attention_tq merge");
    b->dispatch_count++;
    return LC_OK;
}

}  // namespace

extern "C" {

int lc_flash_attention_tq_into(lc_kernels *k, lc_batch *b, const lc_buf *rq, const lc_buf *k_codes,
                               const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                               const lc_buf *levels, lc_buf *out, uint32_t head_dim, uint32_t kv_len,
                               uint32_t current_pos, uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window,
                               uint32_t bits, uint32_t ring_capacity, float softmax_scale) {
    return tq_attention("flash_attention_tq", k, b, rq, false, k_codes, k_norms, v_codes, v_norms, levels, nullptr,
                        out, nullptr, head_dim, kv_len, current_pos, 0, num_q_heads, num_kv_heads, window, bits, 1,
                        ring_capacity, softmax_scale);
}

int lc_flash_attention_tq_batched_into(lc_kernels *k, lc_batch *b, const lc_buf *rq, const lc_buf *k_codes,
                                       const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                                       const lc_buf *levels, lc_buf *out, const lc_buf *positions,
                                       uint32_t head_dim, uint32_t lane_capacity, uint32_t num_q_heads,
                                       uint32_t num_kv_heads, uint32_t window, uint32_t bits, uint32_t n_lanes,
                                       uint32_t ring_capacity, float softmax_scale) {
    if (!positions) return lc_fail(LC_ERR_INVALID_ARGUMENT, "flash_attention_tq_batched: positions is NULL");
    return tq_attention("flash_attention_tq_batched", k, b, rq, false, k_codes, k_norms, v_codes, v_norms, levels,
                        nullptr, out, positions, head_dim, 0, 0, lane_capacity, num_q_heads, num_kv_heads, window,
                        bits, n_lanes, ring_capacity, softmax_scale);
}

int lc_tq_attention_into(lc_kernels *k, lc_batch *b, const lc_buf *q, const lc_buf *k_codes, const lc_buf *k_norms,
                         const lc_buf *v_codes, const lc_buf *v_norms, const lc_buf *levels, const lc_buf *signs,
                         lc_buf *attn_out, uint32_t head_dim, uint32_t kv_len, uint32_t current_pos,
                         uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window, uint32_t bits,
                         uint32_t ring_capacity, float softmax_scale) {
    return tq_attention("tq_attention", k, b, q, true, k_codes, k_norms, v_codes, v_norms, levels, signs, attn_out,
                        nullptr, head_dim, kv_len, current_pos, 0, num_q_heads, num_kv_heads, window, bits, 1,
                        ring_capacity, softmax_scale);
}

// Prefill / multi-row verify over codes (shaders/attention_flash_tq.metal:290-556, kernels.rs:5259-5420): row r of the
// chunk is a decode query at position start_pos + r over the one cache that already holds the chunk's rows.  Here both
// reference kernels map onto the same launch: the prefill kernel (attention_tq_pf.cu) for chunks that pay for it, else the
// decode kernels with the chunk's rows as the grid's third dimension.  The "tiled" entry point keeps the reference's name
// and argument list so callers can switch either way.
int lc_flash_attention_tq_prefill_into(lc_kernels *k, lc_batch *b, const lc_buf *rq, const lc_buf *k_codes,
                                       const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                                       const lc_buf *levels, lc_buf *out, uint32_t head_dim, uint32_t kv_len,
                                       uint32_t start_pos, uint32_t n_rows, uint32_t num_q_heads, uint32_t num_kv_heads,
                                       uint32_t window, uint32_t bits, uint32_t ring_capacity, float softmax_scale) {
    if (n_rows == 0) return LC_OK;
    return tq_attention("flash_attention_tq_prefill", k, b, rq, false, k_codes, k_norms, v_codes, v_norms, levels, nullptr,
                        out, nullptr, head_dim, kv_len, start_pos, 0, num_q_heads, num_kv_heads, window, bits, 1,
                        ring_capacity, softmax_scale, n_rows);
}

int lc_flash_attention_tq_prefill_tiled_into(lc_kernels *k, lc_batch *b, const lc_buf *rq, const lc_buf *k_codes,
                                             const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                                             const lc_buf *levels, lc_buf *out, uint32_t head_dim, uint32_t kv_len,
                                             uint32_t start_pos, uint32_t n_rows, uint32_t num_q_heads,
                                             uint32_t num_kv_heads, uint32_t window, uint32_t bits,
                                             uint32_t ring_capacity, float softmax_scale) {
    if (n_rows == 0) return LC_OK;
    return tq_attention("flash_attention_tq_prefill_tiled", k, b, rq, false, k_codes, k_norms, v_codes, v_norms, levels,
                        nullptr, out, nullptr, head_dim, kv_len, start_pos, 0, num_q_heads, num_kv_heads, window, bits, 1,
                        ring_capacity, softmax_scale, n_rows);
}

// The three dispatches QuantizedKvCache::fused_attention_batch_into issues (kv_cache/quant_cache.rs:620-700) in one
// call: q f16 [n_rows, n_q, hd] in, attn_out f16 out.
int lc_tq_attention_prefill_into(lc_kernels *k, lc_batch *b, const lc_buf *q, const lc_buf *k_codes, const lc_buf *k_norms,
                                 const lc_buf *v_codes, const lc_buf *v_norms, const lc_buf *levels, const lc_buf *signs,
                                 lc_buf *attn_out, uint32_t head_dim, uint32_t kv_len, uint32_t start_pos, uint32_t n_rows,
                                 uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window, uint32_t bits,
                                 uint32_t ring_capacity, float softmax_scale) {
    if (n_rows == 0) return LC_OK;
    return tq_attention("tq_attention_prefill", k, b, q, true, k_codes, k_norms, v_codes, v_norms, levels, signs, attn_out,
                        nullptr, head_dim, kv_len, start_pos, 0, num_q_heads, num_kv_heads, window, bits, 1, ring_capacity,
                        softmax_scale, n_rows);
}

int lc_tq_attention_batched_into(lc_kernels *k, lc_batch *b, const lc_buf *q, const lc_buf *k_codes,
                                 const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                                 const lc_buf *levels, const lc_buf *signs, lc_buf *attn_out,
                                 const lc_buf *positions, uint32_t head_dim, uint32_t lane_capacity,
                                 uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window, uint32_t bits,
                                 uint32_t n_lanes, uint32_t ring_capacity, float softmax_scale) {
    if (!positions) return lc_fail(LC_ERR_INVALID_ARGUMENT, "tq_attention_batched: positions is NULL");
    return tq_attention("tq_attention_batched", k, b, q, true, k_codes, k_norms, v_codes, v_norms, levels, signs,
                        attn_out, positions, head_dim, 0, 0, lane_capacity, num_q_heads, num_kv_heads, window, bits,
                        n_lanes, ring_capacity, softmax_scale);
}

}  // extern "C"

bool lc_qfrag_supported(uint32_t head_dim, uint32_t bits, uint32_t n_q_heads, uint32_t n_kv_heads) {
    return head_dim == 256 && bits >= 2 && bits <= 4 && n_kv_heads >= 1 && n_q_heads % n_kv_heads == 0 &&
           (n_q_heads / n_kv_heads) % 8 == 0;
}

int lc_tq_attention_batched_frag(lc_kernels *k, lc_batch *b, const lc_buf *q, const lc_buf *k_codes, const lc_buf *k_norms,
                                 const lc_buf *v_codes, const lc_buf *v_norms, const lc_buf *levels, const lc_buf *signs,
                                 lc_buf *attn_out, const lc_buf *positions, uint32_t head_dim, uint32_t lane_capacity,
                                 uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window, uint32_t bits,
                                 uint32_t n_lanes, uint32_t ring_capacity, float softmax_scale, const lc_buf *qfrag) {
    if (!positions) return lc_fail(LC_ERR_INVALID_ARGUMENT, "tq_attention_batched: positions is NULL");
    return tq_attention("tq_attention_batched", k, b, q, true, k_codes, k_norms, v_codes, v_norms, levels, signs,
                        attn_out, positions, head_dim, 0, 0, lane_capacity, num_q_heads, num_kv_heads, window, bits,
                        n_lanes, ring_capacity, softmax_scale, 0, qfrag);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of lc_tq_attention_into.
//
// Some callers of this library must not allocate device memory at the moment
// they run attention: a serving thread that has handed every spare byte of HBM
// to its KV pool, or a latency-critical loop where cudaMalloc's implicit device
// synchronisation is unacceptable.  The regular
// entry point keeps its split-K partials in a buffer that the `lc_kernels`
// object grows with cudaMalloc on demand; this one keeps them in the fixed
// array below, which is part of the library image: every GPU that loads the
// library holds these 4 MiB until the process exits.
//
// Rules that follow from sharing one array:
//  * the partials of a call must fit: num_q_heads * splits * (head_dim + 2)
//    floats <= LC_NOALLOC_SCRATCH_FLOATS.  The split count is lowered to fit;
//    if even one split does not fit the call is refused with a status.
//  * nothing in the array has to start at zero: every slot the merge kernel
//    reads is written by the split kernel earlier in the same call, so stale
//    contents of the previous call are never observed;
//  * two calls that overlap on the GPU (different streams, or two host threads)
//    race on the array.  Issue them on one stream, or serialise them.
//  * the first call on each device looks up the array's device address
//    (cudaGetSymbolAddress) and, like every launch site of this library, raises
//    the kernels' shared-memory limit on that device; make that first call
//    before any stream capture begins.
//  * this entry point always runs the CUDA-core split kernel, for every head
//    size and bit width; the regular entry point's tensor-core kernel (tq2 at
//    head_dim 256) is not used here, so at that shape it is the slower of the
//    two, with the same results to within the tests' tolerance.
constexpr size_t LC_NOALLOC_SCRATCH_FLOATS = (size_t)1 << 20;  // 4 MiB
static __device__ __align__(256) float g_noalloc_scratch[LC_NOALLOC_SCRATCH_FLOATS];

namespace {

std::atomic<float *> g_noalloc_ptr[LC_MAX_DEVICES];  // device address of g_noalloc_scratch, per device

// The array's name is a host-side stand-in here, not a device address: resolve
// it once per device, with that device current, and leave the caller's current
// device as it was.  Two threads that race on a device's first call both resolve
// the same address, so the slot only needs to be written atomically.
int noalloc_scratch_for(int device, float **out) {
    if (device < 0 || device >= LC_MAX_DEVICES)
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "tq_attention_noalloc: device %d out of range", device);
    float *ptr = g_noalloc_ptr[device].load(std::memory_order_acquire);
    if (!ptr) {
        int prev = -1;
        LC_CUDA_TRY(cudaGetDevice(&prev));
        if (prev != device) LC_CUDA_TRY(cudaSetDevice(device));
        cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_noalloc_scratch);
        if (prev != device) cudaSetDevice(prev);
        if (e != cudaSuccess || !ptr)
            return lc_fail(LC_ERR_CUDA, "tq_attention_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_noalloc_ptr[device].store(ptr, std::memory_order_release);
    }
    *out = ptr;
    return LC_OK;
}

}  // namespace

extern "C" int lc_tq_attention_noalloc_into(lc_batch *b, const lc_buf *q, const lc_buf *k_codes,
                                            const lc_buf *k_norms, const lc_buf *v_codes, const lc_buf *v_norms,
                                            const lc_buf *levels, const lc_buf *signs, lc_buf *attn_out,
                                            uint32_t head_dim, uint32_t kv_len, uint32_t current_pos,
                                            uint32_t num_q_heads, uint32_t num_kv_heads, uint32_t window,
                                            uint32_t bits, uint32_t ring_capacity, float softmax_scale) {
    const char *name = "tq_attention_noalloc";
    if (!b || !q || !k_codes || !k_norms || !v_codes || !v_norms || !levels || !signs || !attn_out)
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: NULL argument", name);
    if (bits < 2 || bits > 4) return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: bits %u not in 2..=4", name, bits);
    if (head_dim != 64 && head_dim != 128 && head_dim != 256 && head_dim != 512)
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: head_dim %u must be 64, 128, 256 or 512", name, head_dim);
    LC_REQUIRE(num_kv_heads >= 1 && num_q_heads >= 1 && num_q_heads % num_kv_heads == 0,
               "%s: num_q_heads %u must be a multiple of num_kv_heads %u", name, num_q_heads, num_kv_heads);
    const size_t cb = (size_t)head_dim * bits / 8, qn = (size_t)num_q_heads * head_dim;
    LC_REQUIRE(q->bytes >= qn * 2 && attn_out->bytes >= qn * 2, "%s: query/output buffers too small", name);
    LC_REQUIRE(levels->bytes >= (4u << bits) && signs->bytes >= head_dim * 4u, "%s: codec buffers too small", name);
    const uint32_t seq_len = kv_len < current_pos + 1 ? kv_len : current_pos + 1;
    const size_t rows = ring_capacity ? (ring_capacity < seq_len ? ring_capacity : seq_len) : seq_len;
    const uint32_t ws = (window > 0 && current_pos + 1 > window) ? current_pos + 1 - window : 0;
    uint32_t len_max = seq_len > ws ? seq_len - ws : 0;
    if (window > 0 && len_max > window) len_max = window;
    LC_REQUIRE(k_codes->bytes >= rows * num_kv_heads * cb && v_codes->bytes >= rows * num_kv_heads * cb &&
                   k_norms->bytes >= rows * num_kv_heads * 2 && v_norms->bytes >= rows * num_kv_heads * 2,
               "%s: KV buffers hold fewer than %zu rows", name, rows);
    LC_REQUIRE(lc_aligned(k_codes->dptr, 16) && lc_aligned(v_codes->dptr, 16),
               "%s: code buffers must be 16-byte aligned", name);

    const size_t per_split = qn / head_dim * (size_t)(head_dim + 2);  // floats of partials per split
    if (per_split > LC_NOALLOC_SCRATCH_FLOATS)
        return lc_fail(LC_ERR_INVALID_ARGUMENT,
                       "%s: %u heads of %u need %zu bytes of partials per split; the built-in scratch holds %zu bytes",
                       name, num_q_heads, head_dim, per_split * sizeof(float), LC_NOALLOC_SCRATCH_FLOATS * sizeof(float));
    float *scratch = nullptr;
    int st = noalloc_scratch_for(b->ctx->device, &scratch);
    if (st != LC_OK) return st;

    const uint32_t group = num_q_heads / num_kv_heads;
    const int g = group > 4 ? 8 : (group > 2 ? 4 : (group > 1 ? 2 : 1));
    const uint32_t gchunks = (group + g - 1) / g;
    const uint32_t base = num_kv_heads * gchunks;
    uint32_t n_splits = (2u * (uint32_t)b->ctx->sm_count + base - 1) / base;
    uint32_t by_len = (len_max + NW * TILE - 1) / (NW * TILE);
    if (by_len < 1) by_len = 1;
    if (n_splits > by_len) n_splits = by_len;
    if (n_splits > 64) n_splits = 64;
    const uint32_t fit = (uint32_t)(LC_NOALLOC_SCRATCH_FLOATS / per_split);
    if (n_splits > fit) n_splits = fit;
    if (n_splits < 1) n_splits = 1;

    TqAttnParams p;
    p.out_f16 = nullptr;
    p.qfrag = nullptr;
    p.early_kv = 0;
    p.cluster_merge = 0;
    p.queue_chunk = 0;
    p.n_lanes = 1;
    p.counters = nullptr;
    p.pf_heads = 1;
    p.wait_limit = 0;
    p.extra_arrivals = 0;
    p.rq = nullptr;
    p.q = (const __half *)q->dptr;
    p.signs = (const float *)signs->dptr;
    p.kc = (const uint8_t *)k_codes->dptr;
    p.vc = (const uint8_t *)v_codes->dptr;
    p.kn = (const __half *)k_norms->dptr;
    p.vn = (const __half *)v_norms->dptr;
    p.levels = (const float *)levels->dptr;
    p.out = nullptr;
    p.partial = scratch;
    p.positions = nullptr;
    p.kv_len = kv_len;
    p.current_pos = current_pos;
    p.row_positions = 0;
    p.lane_capacity = 0;
    p.n_q = num_q_heads;
    p.n_kv = num_kv_heads;
    p.window = window;
    p.ring = ring_capacity;
    p.n_splits = n_splits;
    p.group = group;
    p.fused_q = 1;
    p.direct_out = 0;
    p.scale = softmax_scale;
    p.status = nullptr;
    dim3 grid(n_splits, num_kv_heads * gchunks, 1);
    switch (head_dim) {
        case 64: st = launch_split_b<64>(b, p, grid, g, bits); break;
        case 128: st = launch_split_b<128>(b, p, grid, g, bits); break;
        case 256: st = launch_split_b<256>(b, p, grid, g, bits); break;
        default: st = launch_split_b<512>(b, p, grid, g, bits); break;
    }
    if (st != LC_OK) return st;
    LC_LAUNCH_CHECKED(lc_launch(tq_attn_merge_kernel<true>, dim3(num_q_heads), dim3(merge_threads(head_dim, n_splits)), 0, b, scratch, (const float *)signs->dptr, nullptr,
                                                                       (__half *)attn_out->dptr, head_dim, n_splits, nullptr, num_q_heads, 0u, 0u));
    LC_CHECK_LAUNCH("tq_attention_noalloc merge");
    b->dispatch_count++;
    return LC_OK;
}
