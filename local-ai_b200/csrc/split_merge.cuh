// Merge of many partial results of few attention heads: a cluster of CTAs per head.
//
// With one CTA per head the partials of a head, 1 KB each at head_dim 256, come through one SM: 148 of them are 3300 cycles of its
// share of L2 bandwidth and three rounds of load latency, while all other SMs are idle.  Here every CTA of a cluster of eight
// adds an eighth of a head's splits, all of its loads in flight together, and leaves its sum in the first CTA's shared memory.
// Sums of sums: against 64 bits its error over 32 - 288 splits is 0.65 - 1.10 of the one-CTA order's, 0.92 in the mean, less the more splits.
#pragma once
#include "lc_internal.h"

namespace {

constexpr unsigned MC = 8, MC_THREADS = 256, MC_SPLITS = 32;   // CTAs per head, threads, fewest splits worth it

struct ClusterMerge {
    float red[2 * MC_THREADS];          // [run row][dim]
    float sum[MC_THREADS / 32];
    float slot[MC][512 + 2];            // of the first CTA: what the CTAs of the cluster send, dims, then (max, sum)
    float fwht[512];
};
// ml(s): (max, sum) of split s; acc(s, c): its unnormalised dims 2c, 2c + 1.  True in the first CTA's threads t < hd / 2, which then have
// the head's sums over all n splits (dims 2t, 2t + 1) and their divisor.  Called by all threads; begins with the dependency wait.
template <typename ML, typename ACC>
__device__ __forceinline__ bool cluster_merge(ClusterMerge &sh, unsigned hd, unsigned n, ML &&ml, ACC &&acc, float2 &o, float &gsum) {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");   // awaited before the first store to the first CTA
    const unsigned t = threadIdx.x, lane = t & 31, rank = blockIdx.x % MC;
    const unsigned cols = hd / 2, c = t % cols, r0 = t / cols, rows = MC_THREADS / cols;
    const unsigned s0 = n * rank / MC, s1 = n * (rank + 1) / MC;
    lc_pdl_wait();
    constexpr int AHEAD = 10;
    float2 a[AHEAD], w[AHEAD];
    auto load = [&](unsigned s) {
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            const bool ok = r0 < rows && s + u * rows < s1;
            w[u] = ok ? ml(s + u * rows) : make_float2(-INFINITY, 0.f);
            a[u] = ok ? acc(s + u * rows, c) : make_float2(0.f, 0.f);
        }
    };
    load(s0 + r0);
    float gmax = -INFINITY;
    for (unsigned s = s0 + lane; s < s1; s += 32) gmax = fmaxf(gmax, ml(s).x);
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, i));
    float ps = 0.f;
    float2 po = make_float2(0.f, 0.f);
    for (unsigned s = s0 + r0;; ) {
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            const float f = w[u].x == -INFINITY ? 0.f : expf(w[u].x - gmax);
            ps += f * w[u].y;
            po.x += f * a[u].x;
            po.y += f * a[u].y;
        }
        s += AHEAD * rows;
        if (s >= s1) break;
        load(s);
    }
    if (r0 < rows) {
        *reinterpret_cast<float2 *>(sh.red + r0 * hd + 2 * c) = po;
        if (c == 0) sh.sum[r0] = ps;
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    __syncthreads();
    if (t < cols) {
        for (unsigned r = 1; r < rows; r++) {
            const float2 v = *reinterpret_cast<const float2 *>(sh.red + r * hd + 2 * c);
            po.x += v.x;
            po.y += v.y;
            ps += sh.sum[r];
        }
        auto send = [&](const float *at, float x, float y) {
            uint32_t ra;
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(ra) : "r"((uint32_t)__cvta_generic_to_shared(at)));
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(ra), "f"(x), "f"(y) : "memory");
        };
        send(sh.slot[rank] + 2 * c, po.x, po.y);
        if (c == 0) send(sh.slot[rank] + 512, gmax, ps);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (rank != 0 || t >= cols) return false;
    float all = -INFINITY;
#pragma unroll
    for (unsigned i = 0; i < MC; i++) all = fmaxf(all, sh.slot[i][512]);
    o = make_float2(0.f, 0.f);
    gsum = 0.f;
#pragma unroll
    for (unsigned i = 0; i < MC; i++) {
        const float m = sh.slot[i][512], f = m == -INFINITY ? 0.f : expf(m - all);
        const float2 v = *reinterpret_cast<const float2 *>(sh.slot[i] + 2 * t);
        gsum += f * sh.slot[i][513];
        o.x += f * v.x;
        o.y += f * v.y;
    }
    return true;
}
template <typename... KArgs, typename... Args>
cudaError_t launch_cluster_merge(void (*kern)(KArgs...), unsigned heads, lc_batch *b, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(heads * MC);
    cfg.blockDim = dim3(MC_THREADS);
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = MC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    LcPlain plain(b);
    cfg.attrs = attr;
    cfg.numAttrs = b->ctx->pdl && !plain.serial ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
// Whether a merge of `n` splits of `heads` heads is one for it.  Few heads: all CTAs have an SM each (16384 keys, cluster against one CTA a head:
// 16 heads 13.1 / 16.5 us with the launch before it; 32 heads 16.7 / 15.7, and 19.5 / 18.3 over f16 rows).  Many splits: at 16 of them the cluster's
// start and its two barriers cost what it saves (2000 keys of f16 rows 8.8 / 8.6 us), from 32 on it gains (9000 codes at head_dim 128: 10.8 / 11.1).
inline bool cluster_merge_fits(const lc_ctx *ctx, unsigned heads, unsigned n, unsigned hd) {
    return n >= MC_SPLITS && heads * MC <= (unsigned)ctx->sm_count && (hd == 64 || hd == 128 || hd == 256 || hd == 512);
}

}  // namespace
