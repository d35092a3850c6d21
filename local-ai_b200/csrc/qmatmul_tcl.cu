// Large-batch quantized matmul on tcgen05: C[m, n] = A[m, K] (f16) x W[n, K]^T, W in GGUF Q4_0 / TQ2_0 blocks, any m, meant for
// m > 64 (prefill chunks, decode batches past one MMA tile).  Stands in for the reference's simdgroup-matrix kernels
// matmul_nt_{q4_0,tq2_0}_mma (shaders/matvec_quant.metal:447-577) at those sizes.
//
// A CTA computes 128 weight rows (the MMA's M) x NB <= 128 batch rows (its N) over a range of K, in steps that fill one weight
// slot of 128 tensor-memory columns: 256 k of TQ2_0, or 128 k of Q4_0 as two f16 operands (the rounded weight and what the
// rounding dropped; their MMAs add up to the product with the exact weight).
//   * two warps bring in the raw blocks of each step with 16-byte cp.async (rows are only 2-byte aligned: the enclosing
//     16-byte range) into a ring of four slots.  (A bulk copy per row and step is too small for the copy engine: 128 of them
//     took 9000 cycles.);
//   * two groups of eight warps take alternate steps and turn raw blocks into f16 weights in the group's own slot of tensor
//     memory (tcgen05.st; the MMA reads its A operand there, so the weights never pass through shared memory again);
//   * one thread requests the step's activations, TMA boxes of 64 k x NB rows with the 128-byte swizzle;
//   * two issuing threads, an accumulator of NB columns each, take alternate K = 16 slices and commit to the step's barrier.
// Tensor memory: 2 x 128 accumulator columns + 2 x 128 weight columns.  Everything but the activations is independent of the
// previous kernel and starts before the dependency wait.  Small outputs split K over a thread-block cluster; the partial tiles
// are exchanged through distributed shared memory and added in split order (deterministic).
//
// What bounds it: a step's MMAs take 16 x 64 cycles at NB = 128, its stores into tensor memory about 900; the kernel this one
// replaced unpacked through shared memory, ran every Q4_0 tile in two passes and reached 10 % of the tensor peak.
// Every wait is bounded; on expiry the CTA records a status word and leaves.
#include <stdlib.h>

#include "lc_internal.h"
#include "tcgen05_util.cuh"
#include "tensor_map.h"

namespace {

constexpr int FMT_Q4_0 = 0, FMT_TQ2_0 = 1;
constexpr int ROWS = 128;            // weight rows per CTA
constexpr int MAX_NB = 128;
constexpr int KT = 64;               // k per activation tile (128 bytes per row: the swizzle's width)
constexpr int GROUPS = 2, GROUP_WARPS = 8, NDQ = GROUPS * GROUP_WARPS;
constexpr int NISS = 2, NRAW = 2;
constexpr int NT = (NDQ + NRAW + 1 + NISS) * 32;   // + raw loaders, activation loader, issuers
constexpr int A_BASE = NISS * MAX_NB, A_COLS = 128, TMEM_COLS = A_BASE + GROUPS * A_COLS;   // 512
constexpr int RAW_RS = 112;          // bytes per row and step: at most 72 data + 15 skew, rounded up; an odd multiple of 16
constexpr int RAW_SLOTS = 4, RAW_SLOT = ROWS * RAW_RS;
constexpr int NBAR = 4;              // step barriers: more than the steps in flight
constexpr int MAX_MATS = 3, MAX_KS = 8;
constexpr uint32_t WAIT_LIMIT = 1u << 22;

template <int FMT> struct TclFmt;
template <> struct TclFmt<FMT_Q4_0> { static constexpr int step_k = 128, blocks = 4, bytes = 18, elems = 32; };
template <> struct TclFmt<FMT_TQ2_0> { static constexpr int step_k = 256, blocks = 1, bytes = 66, elems = 256; };

struct TclParams {
    const uint8_t *w[MAX_MATS];
    void *out[MAX_MATS];
    int n[MAX_MATS], tile_end[MAX_MATS];
    int ngroups;
    int m, K, nb;          // nb = blocks per weight row
    int NB, m_tiles;       // batch rows per CTA (multiple of 16); grid.y
    int ks, sps, steps;    // K splits (grid.z, cluster), steps per split, steps of the whole K
    int b_slots;           // activation ring depth, in steps
    int *status;
    uint32_t wait_limit;
    uint32_t order;            // LcOrder::flags
    uint32_t extra_arrivals;   // 0; 1 in the expiry self-test: the "weights ready" barriers then expect an arrival nobody makes
};

__device__ __forceinline__ void store_c(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store_c(float *p, float v) { *p = v; }
__device__ __forceinline__ void store_c4(__half *p, float4 v) {
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(p) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}
__device__ __forceinline__ void store_c4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }

template <int FMT, typename OutT, bool ORDERED>
__global__ void __launch_bounds__(NT, 1) qgemm_tcl_kernel(const __grid_constant__ TclParams p, const __grid_constant__ CUtensorMap x_map) {
    using F = TclFmt<FMT>;
    constexpr int BB = F::bytes, STEP_TILES = F::step_k / KT, STEP_BYTES = F::blocks * BB;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // operand tiles start on 1024-byte boundaries
    const int B_TILE = p.NB * KT * 2, B_SLOT = STEP_TILES * B_TILE, BS = p.b_slots;
    uint8_t *b_s = smem;                                                   // [BS][B_SLOT]; reused by the split exchange
    uint8_t *raw = b_s + max(BS * B_SLOT, p.ks > 1 ? ROWS * p.NB * 4 : 0); // [RAW_SLOTS][RAW_SLOT]
    uint64_t *raw_full = reinterpret_cast<uint64_t *>(raw + RAW_SLOTS * RAW_SLOT);   // [RAW_SLOTS]
    uint64_t *raw_empty = raw_full + RAW_SLOTS;
    uint64_t *a_full = raw_empty + RAW_SLOTS;                              // [GROUPS]
    uint64_t *b_full = a_full + GROUPS;                                    // [NBAR]
    uint64_t *step_done = b_full + NBAR;                                   // [NBAR]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(step_done + NBAR);
    volatile uint32_t *abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    lc_order_begin<ORDERED>(p.order);
    int grp = 0;
    while (grp + 1 < p.ngroups && (int)blockIdx.x >= p.tile_end[grp]) grp++;
    const int n0 = ((int)blockIdx.x - (grp ? p.tile_end[grp - 1] : 0)) * ROWS, m0 = (int)blockIdx.y * p.NB;
    const int n_rows = p.n[grp];
    const uint8_t *wmat = p.w[grp];
    const size_t rb = (size_t)p.nb * BB, w_bytes = rb * (size_t)n_rows;
    const int s0 = (int)blockIdx.z * p.sps, n_steps = max(0, min(p.steps, s0 + p.sps) - s0);   // this CTA's steps

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < RAW_SLOTS; i++) {
            mbar_init(smem_u32(&raw_full[i]), 32 * NRAW);
            mbar_init(smem_u32(&raw_empty[i]), GROUP_WARPS);
        }
        for (int i = 0; i < GROUPS; i++) mbar_init(smem_u32(&a_full[i]), GROUP_WARPS + p.extra_arrivals);
        for (int i = 0; i < NBAR; i++) {
            mbar_init(smem_u32(&b_full[i]), 1);
            mbar_init(smem_u32(&step_done[i]), NISS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t idesc = (1u << 4) | ((uint32_t)(p.NB >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);

    if (warp < NDQ) {
        // =========================== dequantizing warps ===========================
        const int group = warp / GROUP_WARPS, wq = warp % GROUP_WARPS;
        const int r = 32 * (wq & 3) + lane, bq = wq >> 2;     // operand row; which half of the step's bytes
        const int row = n0 + r;
        const bool rvalid = row < n_rows;
        const uint32_t ta = tmem_base + ((uint32_t)(32 * (wq & 3)) << 16) + (uint32_t)(A_BASE + group * A_COLS);
        for (int i = group; i < n_steps; i += GROUPS) {
            const int rs = i % RAW_SLOTS;
            if (!mbar_wait_warp(smem_u32(&raw_full[rs]), (uint32_t)((i / RAW_SLOTS) & 1), p.wait_limit, abort_flag)) break;
            const size_t g0 = (size_t)row * rb + (size_t)(s0 + i) * STEP_BYTES;
            const uint32_t ra = smem_u32(raw + rs * RAW_SLOT + r * RAW_RS) + (uint32_t)(g0 & 15);
            // sixteen code bytes, 2-byte aligned: five aligned words, funnel-shifted into place
            auto codes16 = [&](uint32_t a, uint32_t (&cw)[4]) {
                const uint32_t sh = (a & 3u) * 8u, wa = a & ~3u;
                const uint32_t w0 = lds32(wa), w1 = lds32(wa + 4), w2 = lds32(wa + 8), w3 = lds32(wa + 12), w4 = sh ? lds32(wa + 16) : 0u;
                cw[0] = __funnelshift_r(w0, w1, sh);
                cw[1] = __funnelshift_r(w1, w2, sh);
                cw[2] = __funnelshift_r(w2, w3, sh);
                cw[3] = __funnelshift_r(w3, w4, sh);
            };
            auto half_at = [&](uint32_t a) -> __half {
                uint16_t v;
                asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
                return __ushort_as_half(v);
            };
            // the MMAs that read this slot a step of this group ago
            auto slot_free = [&]() -> bool {
                if (i < GROUPS) return true;
                const int u = i - GROUPS;
                if (!mbar_wait_warp(smem_u32(&step_done[u % NBAR]), (uint32_t)((u / NBAR) & 1), p.wait_limit, abort_flag)) return false;
                tc_fence_after();
                return true;
            };
            bool dead = false;
            if constexpr (FMT == FMT_TQ2_0) {
                const __half d = rvalid ? half_at(ra + 64u) : __float2half(0.0f);
                // the four weights a code can mean, (q - 1) d, as a byte table for prmt
                const uint32_t p01 = (uint32_t)__half_as_ushort(__hneg(d));
                const uint32_t p23 = (uint32_t)__half_as_ushort(d) | ((uint32_t)__half_as_ushort(__hadd(d, d)) << 16);
                const uint32_t lut_lo = __byte_perm(p01, p23, 0x6420), lut_hi = __byte_perm(p01, p23, 0x7531);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t cw[4], v[4][8];
                    codes16(ra + (uint32_t)(32 * h + 16 * bq), cw);
#pragma unroll
                    for (int l = 0; l < 4; l++)
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t sel = ((cw[q] >> (2 * l)) & 0x03030303u) * 0x11u + 0x40404040u;
                            v[l][2 * q] = __byte_perm(lut_lo, lut_hi, sel);
                            v[l][2 * q + 1] = __byte_perm(lut_lo, lut_hi, sel >> 16);
                        }
                    if (h == 0 && !slot_free()) { dead = true; break; }
                    // element k = 128 h + 32 l + j is bit pair l of code byte 32 h + j: eight columns from k / 2
#pragma unroll
                    for (int l = 0; l < 4; l++) tmem_st8(ta + (uint32_t)(64 * h + 16 * l + 8 * bq), v[l]);
                }
            } else {
                const __half2 c1032 = __float2half2_rn(1032.0f);
#pragma unroll
                for (int bi = 0; bi < 2; bi++) {
                    const int b = 2 * bq + bi;
                    const bool ok = rvalid && (s0 + i) * F::blocks + b < p.nb;
                    uint32_t cw[4], hi[16], lo[16];
                    codes16(ra + (uint32_t)(b * BB + 2), cw);
                    const __half2 d2 = __half2half2(ok ? half_at(ra + (uint32_t)(b * BB)) : __float2half(0.0f));
                    // byte j: k = j in the low nibble, k = j + 16 in the high one
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int nib = 0; nib < 2; nib++)
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                const uint32_t c = __byte_perm(nib ? cw[q] >> 4 : cw[q], 0u, e ? 0x4342 : 0x4140);
                                const uint32_t u = (c & 0x000F000Fu) | 0x64006400u;                           // 1024 + q
                                const __half2 q8 = __hsub2(*reinterpret_cast<const __half2 *>(&u), c1032);     // q - 8, exact
                                const __half2 w = __hmul2(q8, d2), rem = __hfma2(q8, d2, __hneg2(w));          // rounded weight, remainder
                                hi[8 * nib + 2 * q + e] = *reinterpret_cast<const uint32_t *>(&w);
                                lo[8 * nib + 2 * q + e] = *reinterpret_cast<const uint32_t *>(&rem);
                            }
                    if (bi == 0 && !slot_free()) { dead = true; break; }
                    tmem_st16(ta + (uint32_t)(16 * b), hi);
                    tmem_st16(ta + (uint32_t)(64 + 16 * b), lo);
                }
            }
            if (dead) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&raw_empty[rs]));   // the raw bytes are in registers
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&a_full[group]));
        }
    } else if (warp < NDQ + NRAW) {
        // =========================== raw blocks ===========================
        // piece idx of a step: 16 bytes number idx % 6 of row idx / 6 (six pieces hold 72 bytes at any alignment)
        constexpr int PIECES = 6, PER_LANE = ROWS * PIECES / 32 / NRAW;
        const int w = warp - NDQ;
        size_t off[PER_LANE];   // where the row's bytes of the next step start, in the matrix; past its end for rows that do not exist
        uint32_t dst[PER_LANE];
#pragma unroll
        for (int j = 0; j < PER_LANE; j++) {
            const int idx = (j * NRAW + w) * 32 + lane, r = idx / PIECES, pc = idx - r * PIECES;
            off[j] = n0 + r < n_rows ? (size_t)(n0 + r) * rb + (size_t)s0 * STEP_BYTES : w_bytes;
            dst[j] = smem_u32(raw) + (uint32_t)(r * RAW_RS + pc * 16);
        }
        for (int i = 0; i < n_steps; i++) {
            const int rs = i % RAW_SLOTS;
            if (i >= RAW_SLOTS && !mbar_wait_warp(smem_u32(&raw_empty[rs]), (uint32_t)((i / RAW_SLOTS - 1) & 1), p.wait_limit, abort_flag)) break;
#pragma unroll
            for (int j = 0; j < PER_LANE; j++) {
                const int idx = (j * NRAW + w) * 32 + lane, pc = idx % PIECES;
                const size_t at = (off[j] & ~(size_t)15) + (size_t)(pc * 16);
                const size_t left = at < w_bytes ? w_bytes - at : 0;   // nothing is read past the matrix: the rest is zero-filled
                const uint32_t n = left < 16 ? (uint32_t)left : 16u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst[j] + (uint32_t)(rs * RAW_SLOT)), "l"(wmat + (n ? at : 0)), "r"(n)
                             : "memory");
                off[j] += STEP_BYTES;
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(&raw_full[rs])) : "memory");
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else if (warp == NDQ + NRAW) {
        // =========================== activations (one thread) ===========================
        if (lane == 0) {
            lc_order_wait<ORDERED>(p.order);   // the activations are the predecessor's output
            uint32_t slot = 0;
            for (int i = 0; i < n_steps; i++) {
                if (i >= BS) {   // its slot was last read by the MMAs of step i - BS
                    const int u = i - BS;
                    if (!mbar_wait(smem_u32(&step_done[u % NBAR]), (uint32_t)((u / NBAR) & 1), p.wait_limit) || *abort_flag) { *abort_flag = 1; break; }
                }
                const uint32_t bar = smem_u32(&b_full[i % NBAR]), dst = smem_u32(b_s) + slot * (uint32_t)B_SLOT;
                if (++slot == (uint32_t)BS) slot = 0;
                mbar_expect_tx(bar, (uint32_t)B_SLOT);
#pragma unroll
                for (int t = 0; t < STEP_TILES; t++) tma_load_2d(dst + t * B_TILE, &x_map, (s0 + i) * F::step_k + t * KT, m0, bar);
            }
        }
        __syncwarp();
    } else {
        // =========================== MMA issue (two warps) ===========================
        // The whole warp runs the loop, so that descriptors stay in uniform registers; one lane issues (with a loop of that lane alone
        // 509 x 1536 x 6144 Q4_0 took 27.2 instead of 25.5 us).
        const int iw = warp - NDQ - NRAW - 1;
        const bool leader = elect_one();
        const uint64_t bdesc0 = make_desc(smem_u32(b_s) + (uint32_t)(iw * 32));
        const uint32_t acc = tmem_base + (uint32_t)(iw * MAX_NB), ta0 = tmem_base + (uint32_t)(A_BASE + 8 * iw);
        bool dead = false;
        uint32_t slot = 0;
        for (int i = 0; i < n_steps; i++) {
            const uint32_t sa = (uint32_t)i % GROUPS;
            if (!mbar_wait_warp(smem_u32(&a_full[sa]), (uint32_t)((i / GROUPS) & 1), p.wait_limit, abort_flag) ||
                !mbar_wait_warp(smem_u32(&b_full[i % NBAR]), (uint32_t)((i / NBAR) & 1), p.wait_limit, abort_flag)) { dead = true; break; }
            tc_fence_after();
            const uint32_t ta = ta0 + sa * (uint32_t)A_COLS;
            const uint64_t bd = bdesc0 + (uint64_t)((slot * (uint32_t)B_SLOT) >> 4);
            if (++slot == (uint32_t)BS) slot = 0;
            // K = 16 slices iw, iw + 2, ..: slice s of the step is 32 bytes (s % 4) of activation tile s / 4
            if (leader) {
#pragma unroll
                for (int j = 0; j < STEP_TILES * 2; j++) {
                    const uint64_t bj = bd + (uint64_t)(((uint32_t)((j >> 1) * B_TILE) + (uint32_t)((j & 1) * 64)) >> 4);
                    umma_f16_ta(acc, ta + (uint32_t)(16 * j), bj, idesc, (i > 0 || j > 0) ? 1u : 0u);
                    if (FMT == FMT_Q4_0) umma_f16_ta(acc, ta + (uint32_t)(64 + 16 * j), bj, idesc, 1u);
                }
                umma_commit(smem_u32(&step_done[i % NBAR]));
            }
            __syncwarp();
        }
        if (!dead && n_steps > 0) {   // drain: the last step's barrier completes when both issuers' MMAs are done
            const int last = n_steps - 1;
            dead = !mbar_wait_warp(smem_u32(&step_done[last % NBAR]), (uint32_t)((last / NBAR) & 1), p.wait_limit, abort_flag);
        }
        if (dead) *abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const bool failed = *abort_flag != 0;

    // ---- results.  Dequantizing warp w reads TMEM lanes 32 (w & 3) .. + 31 (one weight row per thread) and every fourth group
    //      of 16 batch columns; the two accumulators are added ----
    float *red = reinterpret_cast<float *>(b_s);   // split exchange: [NB cols][128 rows]
    OutT *out = reinterpret_cast<OutT *>(p.out[grp]);
    if (warp < NDQ) {
        const int lrow = 32 * (warp & 3) + lane;
        for (int c0 = 16 * (warp >> 2); c0 < p.NB; c0 += 64) {
            uint32_t a0[16], a1[16];
            float v[16];
            if (!failed && n_steps > 0) {
                const uint32_t t = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0;
                tmem_ld16(t, a0);
                tmem_ld16(t + MAX_NB, a1);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = __uint_as_float(a0[j]) + __uint_as_float(a1[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = 0.f;
            }
            if (p.ks > 1) {
#pragma unroll
                for (int j = 0; j < 16; j++) red[(c0 + j) * ROWS + lrow] = v[j];
            } else if (n0 + lrow < n_rows && !failed) {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (m0 + c0 + j < p.m) store_c(out + (size_t)(m0 + c0 + j) * n_rows + n0 + lrow, v[j]);
            }
        }
    }
    if (p.ks > 1) {
        // The ks CTAs of this tile are one cluster.  An item is four consecutive output rows of one batch column; CTA `rank`
        // finishes every ks-th run of 32 items: adds the partials in split order and stores.
        cluster_sync();
        const int rank = (int)blockIdx.z, cols = min(p.NB, p.m - m0);
        const uint32_t red_a = smem_u32(red);
        if (!failed) {
            for (int col = rank + p.ks * warp; col < cols; col += p.ks * (NT / 32)) {   // a warp finishes a column: 32 x 4 rows
                const int r4 = lane * 4;
                const uint32_t la = red_a + (uint32_t)((col * ROWS + r4) * 4);
                float4 pv[MAX_KS];
#pragma unroll
                for (int sp = 0; sp < MAX_KS; sp++) pv[sp] = sp < p.ks ? ld_dsmem_f4(la, (uint32_t)sp) : make_float4(0.f, 0.f, 0.f, 0.f);
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int sp = 0; sp < MAX_KS; sp++) {
                    a.x += pv[sp].x; a.y += pv[sp].y; a.z += pv[sp].z; a.w += pv[sp].w;
                }
                OutT *dst = out + (size_t)(m0 + col) * n_rows + n0 + r4;
                if (n0 + r4 + 3 < n_rows && (((uintptr_t)dst) & (4 * sizeof(OutT) - 1)) == 0) {
                    store_c4(dst, a);
                } else {
                    const float e[4] = {a.x, a.y, a.z, a.w};
                    for (int q = 0; q < 4; q++)
                        if (n0 + r4 + q < n_rows) store_c(dst + q, e[q]);
                }
            }
        }
        cluster_sync();   // no CTA leaves while a peer may still read its shared memory
    }
    if (failed) tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, tid);
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    lc_order_end<ORDERED>(p.order);
}

// The activations x[m, K] (f16, row-major): boxes of 64 k x NB rows land as NB rows of 128 bytes with the 128-byte swizzle;
// rows beyond m and k beyond K read as zero.
int make_x_map(CUtensorMap *map, const void *x, uint32_t m, uint32_t kk, uint32_t nb) {
    lc_encode_tiled_fn fn = lc_encode_tiled();
    if (!fn) return lc_fail(LC_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {kk, m};
    const cuuint64_t strides[1] = {(cuuint64_t)kk * 2};
    const cuuint32_t box[2] = {KT, nb};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return lc_fail(LC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return LC_OK;
}

template <int FMT, typename OutT, bool ORDERED>
int launch_tcl_as(lc_batch *b, bool serial, const TclParams &p, const CUtensorMap &x_map, int tiles, size_t smem) {
    auto kern = qgemm_tcl_kernel<FMT, OutT, ORDERED>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, p.m_tiles, p.ks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (b->ctx->pdl && !serial) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    if (p.ks > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = (unsigned)p.ks;
        na++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    LC_LAUNCH_CHECKED(cudaLaunchKernelEx(&cfg, kern, p, x_map));
    b->dispatch_count++;
    return LC_OK;
}

template <int FMT, typename OutT>
int launch_tcl(lc_batch *b, bool serial, const TclParams &p, const CUtensorMap &x_map, int tiles, size_t smem) {
    return p.order ? launch_tcl_as<FMT, OutT, true>(b, serial, p, x_map, tiles, smem) : launch_tcl_as<FMT, OutT, false>(b, serial, p, x_map, tiles, smem);
}

}  // namespace

// Batch rows per CTA and K splits of a launch of `tiles` 128-row tiles: a step costs its tensor-memory stores (about 900 cycles)
// or its MMAs (8 per column), whichever is more; a launch costs about 2500 cycles around its steps, the exchange of a split 3000
// more.  Clusters cannot use every SM, other launches can.
struct TclPlan {
    int m_tiles, NB, ks, sps, steps;   // ks splits of sps steps
    uint64_t waves;
};
static TclPlan tcl_plan(int fmt, const lc_kernels *k, uint32_t m, uint32_t kk, int tiles) {
    const int step_k = fmt == FMT_Q4_0 ? TclFmt<FMT_Q4_0>::step_k : TclFmt<FMT_TQ2_0>::step_k;
    TclPlan pl = {1, 16, 1, 1, ((int)kk + step_k - 1) / step_k, 1};
    uint64_t best = ~0ull;
    for (int mt = ((int)m + MAX_NB - 1) / MAX_NB; mt <= ((int)m + 47) / 48; mt++) {
        const int nb = (((int)m + mt - 1) / mt + 15) / 16 * 16, real_mt = ((int)m + nb - 1) / nb;
        for (int ks = 1; ks <= MAX_KS && (ks == 1 || 2 * ks <= pl.steps); ks++) {
            const uint64_t at_once = ks > 1 ? k->cluster_cap[ks] : (uint64_t)k->ctx->sm_count, waves = ((uint64_t)tiles * real_mt + at_once - 1) / at_once;
            const uint64_t cost = waves * (2500u + (uint64_t)((pl.steps + ks - 1) / ks) * (uint64_t)(8 * nb > 900 ? 8 * nb : 900) + (ks > 1 ? 3000u + 10u * nb : 0u));
            if (cost < best) {
                best = cost;
                pl.m_tiles = real_mt;
                pl.NB = nb;
                pl.ks = ks;
                pl.waves = waves;
            }
        }
    }
    pl.sps = (pl.steps + pl.ks - 1) / pl.ks;
    pl.ks = (pl.steps + pl.sps - 1) / pl.sps;
    return pl;
}

// What a launch over one Q4_0 matrix takes at 17 .. 64 rows, in ns, for the choice between this kernel and the register-direct one
// (qmatmul_mma.cu) where there are more tiles than SMs; 0 with fewer, where this one is never the slower by more than 1 % (20 x 512 x 6144:
// 5.45 us against 5.41; 24 x 16384 x 256 5.1 / 5.8; 24 x 4096 x 6144 15.4 / 17.4; eight of 24 x 1536 x 512 in one batch 25.8 / 37.7).
// Fitted to n 24000 .. 262144, K 256 .. 1536: a wave costs its start and epilogue and about 720 a step.
uint64_t lc_qgemm_tcl_estimate(const lc_kernels *k, uint32_t m, uint32_t kk, uint32_t n) {
    const uint64_t tiles = (n + ROWS - 1) / ROWS, sms = (uint64_t)k->ctx->sm_count;
    if (tiles <= sms) return 0;
    const TclPlan pl = tcl_plan(FMT_Q4_0, k, m, kk, (int)tiles);
    return pl.waves * (3300 + 720 * (uint64_t)pl.sps);
}

// Grouped launch: `ng` weight matrices [ns[g], kk] sharing the activations `input` [m, kk].  Returns LC_OK after a launch, a
// positive status on error, or -1 when the shape is outside what this kernel covers (the caller then uses the CUDA-core path).
int lc_qgemm_tcl_launch(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                        lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk) {
    if (m < 1 || ng < 1 || ng > MAX_MATS || !lc_aligned(input->dptr, 16) || kk % 8 != 0) return -1;
    TclParams p;
    p.m = (int)m;
    p.K = (int)kk;
    p.nb = fmt == FMT_Q4_0 ? (int)(kk / 32) : (int)(kk / 256);
    p.ngroups = ng;
    int tiles = 0;
    for (int g = 0; g < MAX_MATS; g++) {
        const int gi = g < ng ? g : ng - 1;
        if (!lc_aligned(weights[gi]->dptr, 16)) return -1;
        p.w[g] = (const uint8_t *)weights[gi]->dptr;
        p.out[g] = outputs[gi]->dptr;
        p.n[g] = (int)ns[gi];
        if (g < ng) tiles += ((int)ns[g] + ROWS - 1) / ROWS;
        p.tile_end[g] = tiles;
    }
    if (tiles < 1) return -1;
    const int step_k = fmt == FMT_Q4_0 ? TclFmt<FMT_Q4_0>::step_k : TclFmt<FMT_TQ2_0>::step_k;
    const TclPlan pl = tcl_plan(fmt, k, m, kk, tiles);
    p.steps = pl.steps;
    p.m_tiles = pl.m_tiles;
    p.NB = pl.NB;
    p.ks = pl.ks;
    p.sps = pl.sps;
    if (p.m_tiles > 65535) return -1;
    p.status = k->dev_status;
    p.wait_limit = k->test_wait_expiry ? 4096u : WAIT_LIMIT;
    p.extra_arrivals = k->test_wait_expiry ? 1u : 0u;
    const size_t b_slot = (size_t)(step_k / KT) * p.NB * KT * 2, fixed = (size_t)RAW_SLOTS * RAW_SLOT + 256 + 1024;
    p.b_slots = (int)((220 * 1024 - fixed) / b_slot);
    if (p.b_slots > NBAR) p.b_slots = NBAR;
    if (p.b_slots > p.sps) p.b_slots = p.sps;
    size_t b_bytes = b_slot * p.b_slots;
    if (p.ks > 1 && b_bytes < (size_t)ROWS * p.NB * 4) b_bytes = (size_t)ROWS * p.NB * 4;
    const size_t smem = fixed + b_bytes;
    if (smem > k->ctx->smem_optin) return -1;
    CUtensorMap x_map;
    int st = make_x_map(&x_map, input->dptr, m, kk, (uint32_t)p.NB);
    if (st != LC_OK) return st;
    size_t w_bytes[MAX_MATS], out_bytes[MAX_MATS];
    for (int g = 0; g < ng; g++) {
        w_bytes[g] = (size_t)p.nb * (fmt == FMT_Q4_0 ? 18 : 66) * ns[g];
        out_bytes[g] = (size_t)m * ns[g] * (f32out ? 4 : 2);
    }
    LcOrder order(b, input, (size_t)m * kk * 2, ng, weights, w_bytes, outputs, out_bytes);
    p.order = order.flags;
    if (fmt == FMT_Q4_0)
        st = f32out ? launch_tcl<FMT_Q4_0, float>(b, order.serial, p, x_map, tiles, smem) : launch_tcl<FMT_Q4_0, __half>(b, order.serial, p, x_map, tiles, smem);
    else
        st = f32out ? launch_tcl<FMT_TQ2_0, float>(b, order.serial, p, x_map, tiles, smem) : launch_tcl<FMT_TQ2_0, __half>(b, order.serial, p, x_map, tiles, smem);
    order.launched = st == LC_OK;
    return st;
}
