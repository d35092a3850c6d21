// FP16-KV decode attention: the three kernels the reference keeps beside the
// code-space path.  Stands in for shaders/flash_decoding.metal:10-189
// (flash_decoding_split / _reduce), shaders/attention_flash.metal:398-503
// (flash_attention_windowed_split) and shaders/attention_sliding.metal:18-78.
// All three are the same computation — softmax(q.K^T * scale) V over the keys
// t in [max(0, pos+1-window), min(kv_len, pos+1)) of one query position — so
// they share one split-K kernel and one merge kernel here; they differ only in
// who owns the partial buffers and how the split count is chosen.
// K/V are f16 [kv_len, n_kv, hd]; q and output are f16 [n_q, hd].
#include <math.h>

#include "lc_internal.h"
#include "split_merge.cuh"

namespace {

constexpr int NT = 256;
constexpr int NW = NT / 32;
constexpr int MAX_DPL2 = 8;  // half2 pairs per lane: head_dim <= 512

// grid = (num_splits, n_q). Split s owns a contiguous run of keys; the 8 warps
// stripe it; lane owns dims {2*lane + 64*i, +1}.
__global__ void __launch_bounds__(NT)
f16_attn_split_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                      float *__restrict__ pmax, float *__restrict__ psum, float *__restrict__ pacc, unsigned hd,
                      unsigned kv_len, unsigned current_pos, unsigned n_q, unsigned n_kv, unsigned window,
                      unsigned num_splits, float scale) {
    lc_pdl_trigger();  // successors may be scheduled; they wait for this grid before reading its output
    lc_pdl_wait();     // everything below may read what the predecessor wrote
    __shared__ float m_s[NW], l_s[NW];
    __shared__ float acc_s[NW][512];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned split = blockIdx.x, qh = blockIdx.y;
    const unsigned kvh = qh / (n_q / n_kv);
    const unsigned seq_len = min(kv_len, current_pos + 1u);
    const unsigned win_start = (window > 0u && current_pos + 1u > window) ? current_pos + 1u - window : 0u;
    const unsigned n_keys = seq_len > win_start ? seq_len - win_start : 0u;
    const unsigned per = (n_keys + num_splits - 1) / num_splits;
    const unsigned begin = win_start + split * per;
    const unsigned end = min(seq_len, begin + per);
    const int dpl2 = (int)hd / 64;  // hd is a multiple of 64

    float2 qr[MAX_DPL2], acc[MAX_DPL2];
#pragma unroll
    for (int i = 0; i < MAX_DPL2; i++) {
        acc[i] = make_float2(0.f, 0.f);
        qr[i] = make_float2(0.f, 0.f);
        if (i < dpl2) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(q + (size_t)qh * hd + 2 * lane + 64 * i));
            qr[i] = make_float2(f.x * scale, f.y * scale);
        }
    }
    float m_run = -INFINITY, l_run = 0.f;
    for (unsigned t = begin + warp; t < end; t += NW) {
        const __half *kr = k + ((size_t)t * n_kv + kvh) * hd;
        const __half *vr = v + ((size_t)t * n_kv + kvh) * hd;
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < MAX_DPL2; i++)
            if (i < dpl2) {
                const float2 kf = __half22float2(__ldg(reinterpret_cast<const __half2 *>(kr + 2 * lane + 64 * i)));
                dot = fmaf(qr[i].x, kf.x, dot);
                dot = fmaf(qr[i].y, kf.y, dot);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float m_new = fmaxf(m_run, dot);
        const float rescale = expf(m_run - m_new);
        const float w = expf(dot - m_new);
        l_run = l_run * rescale + w;
        m_run = m_new;
#pragma unroll
        for (int i = 0; i < MAX_DPL2; i++)
            if (i < dpl2) {
                const float2 vf = __half22float2(__ldg(reinterpret_cast<const __half2 *>(vr + 2 * lane + 64 * i)));
                acc[i].x = fmaf(w, vf.x, acc[i].x * rescale);
                acc[i].y = fmaf(w, vf.y, acc[i].y * rescale);
            }
    }
    if (lane == 0) {
        m_s[warp] = m_run;
        l_s[warp] = l_run;
    }
#pragma unroll
    for (int i = 0; i < MAX_DPL2; i++)
        if (i < dpl2) {
            acc_s[warp][2 * lane + 64 * i] = acc[i].x;
            acc_s[warp][2 * lane + 64 * i + 1] = acc[i].y;
        }
    __syncthreads();
    float gmax = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; w++) gmax = fmaxf(gmax, m_s[w]);
    const size_t pi = (size_t)qh * num_splits + split;
    for (unsigned d = threadIdx.x; d < hd; d += NT) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float f = (m_s[w] == -INFINITY) ? 0.f : expf(m_s[w] - gmax);
            o += f * acc_s[w][d];
        }
        pacc[pi * hd + d] = o;
    }
    if (threadIdx.x == 0) {
        float gsum = 0.f;
        for (int w = 0; w < NW; w++) {
            const float f = (m_s[w] == -INFINITY) ? 0.f : expf(m_s[w] - gmax);
            gsum += f * l_s[w];
        }
        pmax[pi] = gmax;
        psum[pi] = gsum;
    }
}

// Tensor-core form for head_dim 64 / 128 / 256 / 512: one CTA serves up to 8 q-heads of a kv-head, so K and V are read once
// per group instead of once per q-head (8191 keys, 8 q-heads on 2 kv-heads of 256: 67 MB of L2 reads became 17 MB,
// 37.7 -> 10.5 us).  Each warp takes 16-key tiles: S^T[16 keys x 8 heads] = K . Q^T with K fragments from ldmatrix,
// O^T[HD x 8 heads] += V^T . P with V fragments from ldmatrix.trans and P as an f16 and the f16 of its remainder (P was
// f32 before and keeps its precision).  K and V tiles alternate in a per-warp cp.async ring of three slots.
template <int HD_>
struct F16Cfg {
    static constexpr int HD = HD_, NW = HD == 512 ? 4 : 8, NT = NW * 32, NS = HD / 16;
    static constexpr int RS = HD * 2 + 16;          // padded row: ldmatrix reads eight rows without bank conflicts
    static constexpr int SLOT = 16 * RS, SLOTS = 3;
    static constexpr int ACC = NW * NS * 4 * 32 * 4;   // warp merge, reuses the ring
    static constexpr int RING = NW * SLOTS * SLOT;
    static constexpr int SMEM = RING > ACC ? RING : ACC;
};
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ void split_h2(float x, float y, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// grid = (num_splits, n_kv * head chunks)
template <typename C>
__global__ void __launch_bounds__(C::NT)
f16_attn_mma_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                    float *__restrict__ pmax, float *__restrict__ psum, float *__restrict__ pacc, unsigned kv_len,
                    unsigned current_pos, unsigned n_q, unsigned n_kv, unsigned window, unsigned num_splits, float scale) {
    constexpr int HD = C::HD, NW = C::NW, NS = C::NS;
    lc_pdl_trigger();
    lc_pdl_wait();
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float m_s[NW][8], l_s[NW][8], f_s[NW][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const unsigned split = blockIdx.x, group = n_q / n_kv, chunks = (group + 7) / 8;
    const unsigned kvh = blockIdx.y / chunks, chunk = blockIdx.y - kvh * chunks;
    const unsigned qh0 = kvh * group + chunk * 8;
    const int gvalid = min(8, (int)(group - chunk * 8));
    const unsigned seq_len = min(kv_len, current_pos + 1u);
    const unsigned win_start = (window > 0u && current_pos + 1u > window) ? current_pos + 1u - window : 0u;
    const unsigned n_keys = seq_len > win_start ? seq_len - win_start : 0u;
    const unsigned per = (n_keys + num_splits - 1) / num_splits;
    const unsigned begin = win_start + split * per;
    const unsigned end = min(seq_len, begin + per);

    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)(warp * C::SLOTS) * C::SLOT;
    auto issue = [&](unsigned u) {   // sub-tile u of this warp: K (even) or V (odd) rows of tile u / 2
        const unsigned t0 = begin + (unsigned)warp * 16u + (u >> 1) * (NW * 16u);
        if (t0 < end) {
            const __half *src = (u & 1) ? v : k;
            const uint32_t dst = ring + (u % C::SLOTS) * C::SLOT;
            constexpr int CPR = HD / 8;   // 16-byte pieces per row
#pragma unroll
            for (int i = 0; i < CPR / 2; i++) {
                const unsigned c = (unsigned)(i * 32 + lane), row = c / CPR, off = c % CPR;
                const unsigned key = min(t0 + row, end - 1u);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + row * C::RS + off * 16u),
                             "l"(src + ((size_t)key * n_kv + kvh) * HD + off * 8u)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(0);
    issue(1);
    uint32_t bq[NS][2];   // head g, dims 16 s + 2t, + 1 and + 8, + 9
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const uint32_t *row = reinterpret_cast<const uint32_t *>(q + (size_t)(qh0 + (g < gvalid ? g : 0)) * HD + 16 * s + 2 * t);
        bq[s][0] = g < gvalid ? row[0] : 0u;
        bq[s][1] = g < gvalid ? row[4] : 0u;
    }
    float o[NS][4];
#pragma unroll
    for (int s = 0; s < NS; s++) o[s][0] = o[s][1] = o[s][2] = o[s][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_part[2] = {0.f, 0.f};   // heads 2t, 2t + 1
    const uint32_t k_lane = (uint32_t)((lane & 15) * C::RS + (lane >> 4) * 16);
    const uint32_t v_lane = (uint32_t)(((lane & 7) + (lane >> 4) * 8) * C::RS + ((lane >> 3) & 1) * 16);
    unsigned u = 0;
    for (unsigned t0 = begin + warp * 16; t0 < end; t0 += NW * 16, u += 2) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();
        const uint32_t ks = ring + (u % C::SLOTS) * C::SLOT + k_lane;
        issue(u + 2);
        float c2[2][4] = {};
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint32_t a[4];
            ldsm4(a, ks + s * 32);
            mma16816(c2[s & 1], a, bq[s][0], bq[s][1]);
        }
        // logits of keys g (row 0) and g + 8 (row 1), heads 2t, 2t + 1
        float p[2][2], resc[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float s0 = t0 + g < end ? (c2[0][h] + c2[1][h]) * scale : -INFINITY;
            const float s1 = t0 + g + 8 < end ? (c2[0][2 + h] + c2[1][2 + h]) * scale : -INFINITY;
            float tm = fmaxf(s0, s1);
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 4));
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 8));
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 16));
            const float m_new = fmaxf(m_run[h], tm);   // finite: key t0 is valid
            resc[h] = expf(m_run[h] - m_new);
            p[0][h] = expf(s0 - m_new);
            p[1][h] = expf(s1 - m_new);
            l_part[h] = l_part[h] * resc[h] + p[0][h] + p[1][h];
            m_run[h] = m_new;
        }
        if (__any_sync(0xffffffffu, resc[0] != 1.0f || resc[1] != 1.0f)) {
#pragma unroll
            for (int s = 0; s < NS; s++) {
                o[s][0] *= resc[0]; o[s][1] *= resc[1]; o[s][2] *= resc[0]; o[s][3] *= resc[1];
            }
        }
        uint32_t bp[2], bl[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint32_t hi, lo;
            split_h2(p[r][0], p[r][1], hi, lo);
            bp[r] = movmatrix_trans(hi);
            bl[r] = movmatrix_trans(lo);
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();
        const uint32_t vs = ring + ((u + 1) % C::SLOTS) * C::SLOT + v_lane;
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint32_t a[4];
            ldsm4t(a, vs + s * 32);
            mma16816(o[s], a, bp[0], bp[1]);
            mma16816(o[s], a, bl[0], bl[1]);
        }
        __syncwarp();   // every lane is done with the K slot of this tile, which takes V rows of the next
        issue(u + 3);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; h++) {
        l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 4);
        l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 8);
        l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 16);
    }
    __syncthreads();
    float *acc = reinterpret_cast<float *>(smem);   // [NW][NS][4][32 lanes]
    if (g == 0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            m_s[warp][2 * t + h] = m_run[h];
            l_s[warp][2 * t + h] = l_part[h];
        }
    }
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[((warp * NS + s) * 4 + j) * 32 + lane] = o[s][j];
    __syncthreads();
    if (threadIdx.x < 8) {
        const int h = threadIdx.x;
        float gmax = -INFINITY, gsum = 0.f;
#pragma unroll
        for (int w = 0; w < NW; w++) gmax = fmaxf(gmax, m_s[w][h]);
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float f = (m_s[w][h] == -INFINITY) ? 0.f : expf(m_s[w][h] - gmax);
            f_s[w][h] = f;
            gsum += f * l_s[w][h];
        }
        if (h < gvalid) {
            pmax[(size_t)(qh0 + h) * num_splits + split] = gmax;
            psum[(size_t)(qh0 + h) * num_splits + split] = gsum;
        }
    }
    __syncthreads();
    // element j of tile s: head 2t + (j & 1), dim 16 s + g + 8 (j >> 1)
    for (int s = warp; s < NS; s += NW)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int h = 2 * t + (j & 1), d = 16 * s + g + 8 * (j >> 1);
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < NW; w++) sum += f_s[w][h] * acc[((w * NS + s) * 4 + j) * 32 + lane];
            if (h < gvalid) pacc[((size_t)(qh0 + h) * num_splits + split) * HD + d] = sum;
        }
}

// flash_decoding.metal:120-189: LSE merge of the partials, f16 store. grid = n_q, block = hd / 2 threads per row of splits:
// thread (column pair c, row r) adds splits r, r + rows, ... with eight loads in flight, the rows meet in shared memory.
__global__ void __launch_bounds__(1024)
f16_attn_reduce_kernel(const float *__restrict__ pmax, const float *__restrict__ psum, const float *__restrict__ pacc,
                       __half *__restrict__ out, unsigned hd, unsigned num_splits) {
    lc_pdl_trigger();  // successors may be scheduled; they wait for this grid before reading its output
    lc_pdl_wait();     // everything below may read what the predecessor wrote
    __shared__ float red[2048], w_s[32], sum_s[32];
    const unsigned qh = blockIdx.x, cols = hd / 2, c = threadIdx.x % cols, r = threadIdx.x / cols, rows = blockDim.x / cols;
    const float *pm = pmax + (size_t)qh * num_splits, *ps = psum + (size_t)qh * num_splits;
    const float *pa = pacc + (size_t)qh * num_splits * hd + 2 * c;
    const bool pairs = (reinterpret_cast<uintptr_t>(pacc) & 7) == 0;   // the caller's buffer may start at any float
    float gmax = -INFINITY;
    for (unsigned s = threadIdx.x; s < num_splits; s += blockDim.x) gmax = fmaxf(gmax, pm[s]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    if ((threadIdx.x & 31) == 0) w_s[threadIdx.x >> 5] = gmax;
    __syncthreads();
    for (unsigned w = 0; w < (blockDim.x + 31) / 32; w++) gmax = fmaxf(gmax, w_s[w]);
    float gsum = 0.f;
    float2 o = make_float2(0.f, 0.f);
    for (unsigned s0 = r; s0 < num_splits; s0 += rows * 8) {
        float2 a[8];
        float m[8], l[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const unsigned s = s0 + i * rows;
            const bool ok = s < num_splits;
            const float *at = pa + (size_t)s * hd;
            a[i] = !ok ? make_float2(0.f, 0.f) : pairs ? *reinterpret_cast<const float2 *>(at) : make_float2(at[0], at[1]);
            m[i] = ok ? pm[s] : -INFINITY;
            l[i] = ok ? ps[s] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float f = m[i] == -INFINITY ? 0.f : expf(m[i] - gmax);
            gsum += f * l[i];
            o.x += f * a[i].x;
            o.y += f * a[i].y;
        }
    }
    *reinterpret_cast<float2 *>(red + r * hd + 2 * c) = o;
    if (c == 0) sum_s[r] = gsum;
    __syncthreads();
    for (unsigned d = threadIdx.x; d < hd; d += blockDim.x) {
        float sum = 0.f, l = 0.f;
        for (unsigned i = 0; i < rows; i++) {
            sum += red[i * hd + d];
            l += sum_s[i];
        }
        out[(size_t)qh * hd + d] = __float2half_rn(l > 0.f ? sum * (1.f / l) : 0.f);
    }
}

// The same with a cluster of CTAs per head (split_merge.cuh): many splits, few heads.  8191 keys, 64 splits of 8 heads: 10.4 -> 9.2 us with
// the launch before it.
__global__ void __launch_bounds__(MC_THREADS)
f16_attn_reduce_cluster_kernel(const float *__restrict__ pmax, const float *__restrict__ psum, const float *__restrict__ pacc,
                               __half *__restrict__ out, unsigned hd, unsigned num_splits) {
    lc_pdl_trigger();
    __shared__ ClusterMerge sh;
    const size_t qh = blockIdx.x / MC;
    const float *pm = pmax + qh * num_splits, *ps = psum + qh * num_splits, *pa = pacc + qh * num_splits * hd;
    const bool pairs = (reinterpret_cast<uintptr_t>(pacc) & 7) == 0;   // the caller's buffer may start at any float
    float2 o;
    float gsum;
    const bool mine = cluster_merge(
        sh, hd, num_splits, [&](unsigned s) { return make_float2(pm[s], ps[s]); },
        [&](unsigned s, unsigned c) {
            const float *at = pa + (size_t)s * hd + 2 * c;
            return pairs ? *reinterpret_cast<const float2 *>(at) : make_float2(at[0], at[1]);
        }, o, gsum);
    if (!mine) return;
    const float inv = gsum > 0.f ? 1.f / gsum : 0.f;
    out[qh * hd + 2 * threadIdx.x] = __float2half_rn(gsum > 0.f ? o.x * inv : 0.f);
    out[qh * hd + 2 * threadIdx.x + 1] = __float2half_rn(gsum > 0.f ? o.y * inv : 0.f);
}

template <int HD>
int launch_mma(lc_batch *b, const __half *q, const __half *k, const __half *v, float *pmax, float *psum, float *pacc, uint32_t kv_len,
               uint32_t current_pos, uint32_t n_q, uint32_t n_kv, uint32_t window, uint32_t num_splits, float scale) {
    using C = F16Cfg<HD>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(f16_attn_mma_kernel<C>, optin, b->ctx, C::SMEM));
    const uint32_t chunks = (n_q / n_kv + 7) / 8;
    LC_LAUNCH_CHECKED(lc_launch(f16_attn_mma_kernel<C>, dim3(num_splits, n_kv * chunks), dim3(C::NT), C::SMEM, b, q, k, v, pmax, psum, pacc,
                                kv_len, current_pos, n_q, n_kv, window, num_splits, scale));
    return LC_OK;
}

// Whether the tensor-core form takes the call: its head sizes, 16-byte loads of K and V rows, 4-byte loads of the query.
bool mma_form(uint32_t hd, const lc_buf *q, const lc_buf *k, const lc_buf *v) {
    return (hd == 64 || hd == 128 || hd == 256 || hd == 512) && lc_aligned(k->dptr, 16) && lc_aligned(v->dptr, 16) && lc_aligned(q->dptr, 4);
}

int f16_attention(const char *name, lc_batch *b, const lc_buf *q, const lc_buf *k, const lc_buf *v, lc_buf *output,
                  float *pmax, float *psum, float *pacc, uint32_t hd, uint32_t kv_len, uint32_t current_pos,
                  uint32_t n_q, uint32_t n_kv, uint32_t window, uint32_t num_splits, float scale) {
    if (!b || !q || !k || !v || !output) return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: NULL argument", name);
    LC_REQUIRE(hd >= 64 && hd <= 512 && hd % 64 == 0, "%s: head_dim %u must be a multiple of 64 up to 512", name, hd);
    LC_REQUIRE(n_kv >= 1 && n_q >= 1 && n_q % n_kv == 0, "%s: num_q_heads %u must be a multiple of num_kv_heads %u",
               name, n_q, n_kv);
    LC_REQUIRE(num_splits >= 1, "%s: num_splits must be >= 1", name);
    const uint32_t seq_len = kv_len < current_pos + 1 ? kv_len : current_pos + 1;
    LC_REQUIRE(q->bytes >= (size_t)n_q * hd * 2 && output->bytes >= (size_t)n_q * hd * 2, "%s: q/output too small", name);
    LC_REQUIRE(k->bytes >= (size_t)seq_len * n_kv * hd * 2 && v->bytes >= (size_t)seq_len * n_kv * hd * 2,
               "%s: K/V hold fewer than %u rows", name, seq_len);
    LC_REQUIRE(lc_aligned(q->dptr, 4) && lc_aligned(k->dptr, 4) && lc_aligned(v->dptr, 4), "%s: buffers must be 4-byte aligned", name);
    const __half *qp = (const __half *)q->dptr, *kp = (const __half *)k->dptr, *vp = (const __half *)v->dptr;
    if (mma_form(hd, q, k, v)) {
        int st;
        switch (hd) {
            case 64: st = launch_mma<64>(b, qp, kp, vp, pmax, psum, pacc, kv_len, current_pos, n_q, n_kv, window, num_splits, scale); break;
            case 128: st = launch_mma<128>(b, qp, kp, vp, pmax, psum, pacc, kv_len, current_pos, n_q, n_kv, window, num_splits, scale); break;
            case 256: st = launch_mma<256>(b, qp, kp, vp, pmax, psum, pacc, kv_len, current_pos, n_q, n_kv, window, num_splits, scale); break;
            default: st = launch_mma<512>(b, qp, kp, vp, pmax, psum, pacc, kv_len, current_pos, n_q, n_kv, window, num_splits, scale); break;
        }
        if (st != LC_OK) return st;
    } else {
        LC_LAUNCH_CHECKED(lc_launch(f16_attn_split_kernel, dim3(num_splits, n_q), dim3(NT), 0, b, qp, kp, vp, pmax, psum, pacc, hd, kv_len,
                                    current_pos, n_q, n_kv, window, num_splits, scale));
    }
    LC_CHECK_LAUNCH(name);
    b->dispatch_count++;
    uint32_t rows = 2048 / hd;   // rows of splits that the block's 1024 threads hold
    if (rows > (num_splits + 7) / 8) rows = (num_splits + 7) / 8;
    if (cluster_merge_fits(b->ctx, n_q, num_splits, hd))
        LC_LAUNCH_CHECKED(launch_cluster_merge(f16_attn_reduce_cluster_kernel, n_q, b, (const float *)pmax, (const float *)psum, (const float *)pacc,
                                               (__half *)output->dptr, hd, num_splits));
    else
        LC_LAUNCH_CHECKED(lc_launch(f16_attn_reduce_kernel, dim3(n_q), dim3(rows * (hd / 2)), 0, b, (const float *)pmax, (const float *)psum,
                                (const float *)pacc, (__half *)output->dptr, hd, num_splits));
    LC_CHECK_LAUNCH(name);
    b->dispatch_count++;
    return LC_OK;
}

// Library-owned partials for the entry points whose reference signature has none.
int f16_attention_scratch(const char *name, lc_kernels *kn, lc_batch *b, const lc_buf *q, const lc_buf *k,
                          const lc_buf *v, lc_buf *output, uint32_t hd, uint32_t kv_len, uint32_t current_pos,
                          uint32_t n_q, uint32_t n_kv, uint32_t window, uint32_t num_splits, float scale) {
    if (!kn) return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: kernels is NULL", name);
    const size_t parts = (size_t)n_q * num_splits;
    int st = lc_reserve_scratch(kn, b, parts * (hd + 2) * sizeof(float), 0);
    if (st != LC_OK) return st;
    float *pmax = (float *)kn->scratch, *psum = pmax + parts, *pacc = psum + parts;
    return f16_attention(name, b, q, k, v, output, pmax, psum, pacc, hd, kv_len, current_pos, n_q, n_kv, window,
                         num_splits, scale);
}

}  // namespace

extern "C" {

uint32_t lc_flash_split_count(const lc_kernels *k, uint32_t eff_seq_len) {
    (void)k;
    const uint32_t c = (eff_seq_len + 15) / 16;  // kernels.rs:1265-1278
    return c < 1 ? 1 : (c > 16 ? 16 : c);
}

int lc_flash_attention_windowed_split_into(lc_kernels *k, lc_batch *b, const lc_buf *q, const lc_buf *kk,
                                           const lc_buf *v, lc_buf *output, lc_buf *partial_max,
                                           lc_buf *partial_sum, lc_buf *partial_acc, uint32_t head_dim,
                                           uint32_t kv_len, uint32_t current_pos, uint32_t num_q_heads,
                                           uint32_t num_kv_heads, uint32_t window, uint32_t num_splits) {
    if (!k || !partial_max || !partial_sum || !partial_acc)
        return lc_fail(LC_ERR_INVALID_ARGUMENT, "flash_attention_windowed_split: NULL argument");
    const size_t parts = (size_t)num_q_heads * num_splits;
    LC_REQUIRE(partial_max->bytes >= parts * 4 && partial_sum->bytes >= parts * 4 &&
                   partial_acc->bytes >= parts * head_dim * 4,
               "flash_attention_windowed_split: partial buffers too small for %u heads x %u splits", num_q_heads,
               num_splits);
    LC_REQUIRE(lc_aligned(partial_max->dptr, 4) && lc_aligned(partial_sum->dptr, 4) && lc_aligned(partial_acc->dptr, 4),
               "flash_attention_windowed_split: partial buffers must be 4-byte aligned");
    return f16_attention("flash_attention_windowed_split", b, q, kk, v, output, (float *)partial_max->dptr,
                         (float *)partial_sum->dptr, (float *)partial_acc->dptr, head_dim, kv_len, current_pos,
                         num_q_heads, num_kv_heads, window, num_splits, 1.0f);
}

int lc_flash_decoding_into(lc_kernels *k, lc_ctx *ctx, lc_batch *b, const lc_buf *q, const lc_buf *kk,
                           const lc_buf *v, lc_buf *output, uint32_t head_dim, uint32_t kv_len, uint32_t current_pos,
                           uint32_t num_q_heads, uint32_t num_kv_heads) {
    (void)ctx;  // the reference needs it to renew the encoder between split and reduce
    const uint32_t seq_len = kv_len < current_pos + 1 ? kv_len : current_pos + 1;
    // The reference splits every 256 keys (FD_SPLIT_SIZE, flash_decoding.metal:12).  Here: one 16-key tile for each of a
    // CTA's eight warps as long as the CTAs fit on the SMs at once (one CTA per SM), then longer splits.
    uint32_t splits = (seq_len + 255) / 256;
    if (k && q && kk && v && num_kv_heads && mma_form(head_dim, q, kk, v)) {
        const uint32_t ctas = num_kv_heads * ((num_q_heads / num_kv_heads + 7) / 8), sms = (uint32_t)k->ctx->sm_count;
        const uint32_t by_len = (seq_len + 127) / 128, fit = ctas < sms ? sms / ctas : 1u;
        splits = by_len < fit ? by_len : fit;
    }
    if (splits < 1) splits = 1;
    return f16_attention_scratch("flash_decoding", k, b, q, kk, v, output, head_dim, kv_len, current_pos,
                                 num_q_heads, num_kv_heads, 0, splits, 1.0f);
}

int lc_attention_sliding(lc_kernels *k, lc_ctx *ctx, const lc_buf *q, const lc_buf *kk, const lc_buf *v,
                         lc_buf *output, uint32_t head_dim, uint32_t kv_len, uint32_t current_pos, uint32_t window,
                         uint32_t num_q_heads, uint32_t num_kv_heads) {
    if (!ctx) return lc_fail(LC_ERR_INVALID_ARGUMENT, "attention_sliding: ctx is NULL");
    const uint32_t seq_len = kv_len < current_pos + 1 ? kv_len : current_pos + 1;
    const uint32_t ws = (window > 0 && current_pos + 1 > window) ? current_pos + 1 - window : 0;
    const uint32_t eff = seq_len > ws ? seq_len - ws : 0;
    // The reference caps the window at its 2048-entry score array
    // (attention_sliding.metal:33); this kernel has no such cap.
    return lc_run_and_wait(ctx, [&](lc_batch *b) {
        return f16_attention_scratch("attention_sliding", k, b, q, kk, v, output, head_dim, kv_len, current_pos,
                                     num_q_heads, num_kv_heads, window, lc_flash_split_count(k, eff), 1.0f);
    });
}

}  // extern "C"
