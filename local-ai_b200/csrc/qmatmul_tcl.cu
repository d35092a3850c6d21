// Large-batch quantized matmul on tcgen05: C[m, n] = A[m, K] (f16) x W[n, K]^T, W in GGUF Q4_0 / TQ2_0 blocks, any m, meant for
// m > 64 (prefill chunks, decode batches past one MMA tile).  Stands in for the reference's simdgroup-matrix kernels
// matmul_nt_{q4_0,tq2_0}_mma (shaders/matvec_quant.metal:447-577) at those sizes.
//
// A CTA computes 128 weight rows (the MMA's M) x NB <= 128 batch rows (its N) over a range of K, in steps that fill one weight
// slot of 64 tensor-memory columns: 128 k of TQ2_0, or 64 k of Q4_0 as two f16 operands (the rounded weight and what the
// rounding dropped; their MMAs add up to the product with the exact weight).
//   * four warps bring in the raw blocks of two steps at a time with 16-byte cp.async (rows are only 2-byte aligned: the enclosing
//     16-byte range) into a ring of four slots, from the kernel's first instruction on.  (A bulk copy per row is too small for the
//     copy engine: 128 of them took 9000 cycles.);
//   * four groups of four warps take a step in turn and turn raw blocks into f16 weights in the group's own slot of tensor
//     memory (tcgen05.st; the MMA reads its A operand there, so the weights never pass through shared memory again);
//   * one thread requests the step's activations, TMA boxes of 64 k x NB rows with the 128-byte swizzle;
//   * two issuing warps, an accumulator of NB columns each, take alternate steps and commit to the step's barrier.
// Tensor memory: 2 x 128 accumulator columns + 4 x 64 weight columns.  Everything but the activations is independent of the
// previous kernel and starts before the dependency wait.  Small outputs split K over a thread-block cluster; the partial tiles
// are exchanged through distributed shared memory and added in split order (deterministic).
//
// What bounds it: 512 x 16384 x 8192 TQ2_0 at 124 us (141 with two raw-block warps, two slots of twice the columns, shifts in place of
// multiplies and results stored from tensor memory), 106 without the conversion, 122 without the MMAs, 127 without the stores into
// tensor memory, 96 without conversion and MMAs: the activations, which every tile of rows fetches from L2, and the conversion's
// integer instructions.  Small launches are bound by their fixed part, some 7000 cycles.
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
constexpr int GROUPS = 4, GROUP_WARPS = 4, NDQ = GROUPS * GROUP_WARPS;
constexpr int NISS = 2, NRAW = 4;
constexpr int NT = (NDQ + NRAW + 1 + NISS) * 32;   // + raw loaders, activation loader, issuers
constexpr int A_BASE = NISS * MAX_NB, A_COLS = 64, TMEM_COLS = A_BASE + GROUPS * A_COLS;   // 512
constexpr int RAW_RS = 112;          // bytes per row and unit of two steps: at most 72 data + 15 skew, rounded up; an odd multiple of 16
constexpr int RAW_SLOTS = 4, RAW_SLOT = ROWS * RAW_RS;
constexpr int NBAR = 8;              // step barriers: more than the steps in flight
constexpr int MAX_MATS = 3, MAX_KS = 8;
constexpr uint32_t WAIT_LIMIT = 1u << 22;

template <int FMT> struct TclFmt;
template <> struct TclFmt<FMT_Q4_0> { static constexpr int step_k = 64, unit_bytes = 4 * 18, block_bytes = 18; };
template <> struct TclFmt<FMT_TQ2_0> { static constexpr int step_k = 128, unit_bytes = 66, block_bytes = 66; };

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

// The raw blocks of a step, by 16-byte cp.async: piece idx is number idx % 6 of row idx / 6 (six pieces hold 72 bytes at any alignment; the
// last is left out where the row's skew lets five hold them).  Four warps and 32-bit addresses: two warps that checked each piece's end
// took 1150 - 1900 cycles for what the rest of the kernel did in 800 (509 x 1536 x 6144 Q4_0 24.7 -> 21.5 us).
template <int FMT>
struct RawLoader {
    static constexpr int UNIT_BYTES = TclFmt<FMT>::unit_bytes, PIECES = 6, PER_LANE = ROWS * PIECES / 32 / NRAW;
    const uint8_t *tile;       // the tile's first row, 16-byte aligned: 128 rows of an even number of bytes
    size_t left;               // bytes from there to the matrix's end
    uint32_t off[PER_LANE];    // where the row's bytes of the next step start
    uint32_t dst[PER_LANE], piece[PER_LANE];
    bool inside;               // no piece reaches past the matrix
    __device__ __forceinline__ void start(const uint8_t *w, size_t rb, int n0, int n_rows, int u0, int n_units, uint32_t raw, int t) {
        tile = w + (size_t)n0 * rb;
        left = (size_t)(n_rows - n0) * rb;
        inside = (((size_t)(ROWS - 1) * rb + (size_t)(u0 + n_units) * UNIT_BYTES + 15) & ~(size_t)15) <= left;
#pragma unroll
        for (int j = 0; j < PER_LANE; j++) {
            const int idx = j * NRAW * 32 + t, r = idx / PIECES, pc = idx - r * PIECES;
            off[j] = (uint32_t)r * (uint32_t)rb + (uint32_t)(u0 * UNIT_BYTES);
            dst[j] = raw + (uint32_t)(r * RAW_RS + pc * 16);
            piece[j] = (uint32_t)(pc * 16);
        }
    }
    __device__ __forceinline__ void unit(int slot, uint32_t bar) {
        const uint32_t at_slot = (uint32_t)(slot * RAW_SLOT);
        if (inside) {
#pragma unroll
            for (int j = 0; j < PER_LANE; j++) {
                if (piece[j] < (off[j] & 15u) + UNIT_BYTES)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst[j] + at_slot), "l"(tile + ((off[j] & ~15u) + piece[j])) : "memory");
                off[j] += UNIT_BYTES;
            }
        } else {
#pragma unroll
            for (int j = 0; j < PER_LANE; j++) {
                const size_t at = (size_t)((off[j] & ~15u) + piece[j]), rest = at < left ? left - at : 0;   // past the matrix: zeros
                const uint32_t n = rest < 16 ? (uint32_t)rest : 16u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst[j] + at_slot), "l"(tile + (n ? at : 0)), "r"(n) : "memory");
                off[j] += UNIT_BYTES;
            }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
    }
};

template <int FMT, typename OutT, bool ORDERED>
__global__ void __launch_bounds__(NT, 1) qgemm_tcl_kernel(const __grid_constant__ TclParams p, const __grid_constant__ CUtensorMap x_map) {
    using F = TclFmt<FMT>;
    constexpr int BB = F::block_bytes, STEP_TILES = F::step_k / KT, UNIT_BYTES = F::unit_bytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // operand tiles start on 1024-byte boundaries
    const int B_TILE = p.NB * KT * 2, B_SLOT = STEP_TILES * B_TILE, BS = p.b_slots;
    uint8_t *b_s = smem;                                                   // [BS][B_SLOT]; reused by the results
    uint8_t *raw = b_s + max(BS * B_SLOT, ROWS * p.NB * 4); // [RAW_SLOTS][RAW_SLOT]
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
    const size_t rb = (size_t)p.nb * BB;
    const int s0 = (int)blockIdx.z * p.sps, n_steps = max(0, min(p.steps, s0 + p.sps) - s0);   // this CTA's steps; s0 is even
    const int u0 = s0 / 2, n_units = (n_steps + 1) / 2;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    const bool raw_warp = warp >= NDQ && warp < NDQ + NRAW;
    RawLoader<FMT> loader;
    if (raw_warp) {   // the first raw blocks leave ahead of everything else; these warps do not wait for the others
        if (tid == NDQ * 32) {
            for (int i = 0; i < RAW_SLOTS; i++) {
                mbar_init(smem_u32(&raw_full[i]), 32 * NRAW);
                mbar_init(smem_u32(&raw_empty[i]), 2 * GROUP_WARPS);
            }
            *abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        asm volatile("bar.sync 1, %0;\n" ::"n"(NRAW * 32) : "memory");
        asm volatile("bar.arrive 2, %0;\n" ::"n"(NT) : "memory");
        loader.start(wmat, rb, n0, n_rows, u0, n_units, smem_u32(raw), tid - NDQ * 32);
    } else {
        if (tid == 0) {
            for (int i = 0; i < GROUPS; i++) mbar_init(smem_u32(&a_full[i]), GROUP_WARPS + p.extra_arrivals);
            for (int i = 0; i < NBAR; i++) {
                mbar_init(smem_u32(&b_full[i]), 1);
                mbar_init(smem_u32(&step_done[i]), 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        tc_fence_before();
        asm volatile("bar.sync 2, %0;\n" ::"n"(NT) : "memory");
        tc_fence_after();
    }
    const uint32_t tmem_base = raw_warp ? 0u : *tmem_slot;
    const uint32_t idesc = (1u << 4) | ((uint32_t)(p.NB >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);

    if (warp < NDQ) {
        // =========================== dequantizing warps ===========================
        const int group = warp / GROUP_WARPS, quarter = warp % GROUP_WARPS, half = group & 1;   // steps group, group + 4, ..: always this half of a unit
        const int r = 32 * quarter + lane;     // operand row
        const int row = n0 + r;
        const bool rvalid = row < n_rows;
        const uint32_t ta = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(A_BASE + group * A_COLS);
        for (int i = group; i < n_steps; i += GROUPS) {
            const int u = i / 2, rs = u % RAW_SLOTS;
            if (!mbar_wait_warp(smem_u32(&raw_full[rs]), (uint32_t)((u / RAW_SLOTS) & 1), p.wait_limit, abort_flag)) break;
            const uint32_t g0 = (uint32_t)r * (uint32_t)rb + (uint32_t)((u0 + u) * UNIT_BYTES);   // (of the tile, which starts on 16 bytes)
            const uint32_t ra = smem_u32(raw + rs * RAW_SLOT + r * RAW_RS) + (g0 & 15u);
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
            // the step is in registers: its raw bytes may go, and the weights go in when the MMAs that read this slot a step of this group ago
            // are done
            bool dead = false;
            auto release = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&raw_empty[rs]));
            };
            auto slot_free = [&]() -> bool {
                if (i < GROUPS) return true;
                const int j = i - GROUPS;
                if (!mbar_wait_warp(smem_u32(&step_done[j % NBAR]), (uint32_t)((j / NBAR) & 1), p.wait_limit, abort_flag)) return false;
                tc_fence_after();
                return true;
            };
            if constexpr (FMT == FMT_TQ2_0) {
                const __half d = rvalid ? half_at(ra + 64u) : __float2half(0.0f);
                // the four weights a code can mean, (q - 1) d, as a byte table for prmt
                const uint32_t p01 = (uint32_t)__half_as_ushort(__hneg(d));
                const uint32_t p23 = (uint32_t)__half_as_ushort(d) | ((uint32_t)__half_as_ushort(__hadd(d, d)) << 16);
                const uint32_t lut_lo = __byte_perm(p01, p23, 0x6420), lut_hi = __byte_perm(p01, p23, 0x7531);
#pragma unroll
                for (int bi = 0; bi < 2; bi++) {
                    uint32_t cw[4], v[4][8];
                    codes16(ra + (uint32_t)(32 * half + 16 * bi), cw);
#pragma unroll
                    for (int l = 0; l < 4; l++)
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t c = (cw[q] >> (2 * l)) & 0x03030303u;
                            uint32_t sel_hi;
                            asm("mad.hi.u32 %0, %1, 0x110000, 0x4040;\n" : "=r"(sel_hi) : "r"(c));
                            v[l][2 * q] = __byte_perm(lut_lo, lut_hi, c * 0x11u + 0x40404040u);
                            v[l][2 * q + 1] = __byte_perm(lut_lo, lut_hi, sel_hi);
                        }
                    if (bi == 0 && !slot_free()) { dead = true; break; }
                    if (bi == 1) release();
#pragma unroll
                    for (int l = 0; l < 4; l++) tmem_st8(ta + (uint32_t)(16 * l + 8 * bi), v[l]);
                }
            } else {
                const __half2 offset[2] = {__float2half2_rn(1032.0f), __float2half2_rn(72.0f)};
#pragma unroll
                for (int bi = 0; bi < 2; bi++) {
                    const int b = 2 * half + bi;
                    const bool ok = rvalid && (u0 + u) * 4 + b < p.nb;
                    uint32_t cw[4], hi[16], lo[16];
                    codes16(ra + (uint32_t)(b * BB + 2), cw);
                    const __half2 d2 = __half2half2(ok ? half_at(ra + (uint32_t)(b * BB)) : __float2half(0.0f));
                    // byte j: k = j in the low nibble, k = j + 16 in the high one; under an exponent in place they are 1024 + q and 64 + q
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const uint32_t c = __byte_perm(cw[q], 0u, e ? 0x4342 : 0x4140);
#pragma unroll
                            for (int nib = 0; nib < 2; nib++) {
                                const uint32_t v = nib ? (c & 0x00F000F0u) | 0x54005400u : (c & 0x000F000Fu) | 0x64006400u;
                                const __half2 q8 = __hsub2(*reinterpret_cast<const __half2 *>(&v), offset[nib]);   // q - 8, exact
                                const __half2 w = __hmul2(q8, d2), rem = __hfma2(q8, d2, __hneg2(w));          // rounded weight, remainder
                                hi[8 * nib + 2 * q + e] = *reinterpret_cast<const uint32_t *>(&w);
                                lo[8 * nib + 2 * q + e] = *reinterpret_cast<const uint32_t *>(&rem);
                            }
                        }
                    if (bi == 0 && !slot_free()) { dead = true; break; }
                    if (bi == 1) release();
                    tmem_st16(ta + (uint32_t)(16 * bi), hi);
                    tmem_st16(ta + (uint32_t)(32 + 16 * bi), lo);
                }
            }
            if (dead) break;
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&a_full[group]));
        }
    } else if (raw_warp) {
        // =========================== raw blocks ===========================
        for (int u = 0; u < n_units; u++) {
            const int rs = u % RAW_SLOTS;
            if (u >= RAW_SLOTS && !mbar_wait_warp(smem_u32(&raw_empty[rs]), (uint32_t)((u / RAW_SLOTS - 1) & 1), p.wait_limit, abort_flag)) break;
            loader.unit(rs, smem_u32(&raw_full[rs]));
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
        const uint64_t bdesc0 = make_desc(smem_u32(b_s));
        const uint32_t acc = tmem_base + (uint32_t)(iw * MAX_NB), ta0 = tmem_base + (uint32_t)A_BASE;
        bool dead = false;
        int slot = iw < BS ? iw : 0;
        for (int i = iw; i < n_steps; i += NISS) {   // every other step, into this warp's accumulator
            const uint32_t sa = (uint32_t)i % GROUPS;
            // (a wait takes some 250 cycles even where its phase is complete; the activations first: 256 x 1536 x 6144 TQ2_0 8.35 -> 8.32 us,
            // 509 x 6144 x 1536 Q4_0 22.75 -> 22.93)
            if (!mbar_wait_warp(smem_u32(&a_full[sa]), (uint32_t)((i / GROUPS) & 1), p.wait_limit, abort_flag) ||
                !mbar_wait_warp(smem_u32(&b_full[i % NBAR]), (uint32_t)((i / NBAR) & 1), p.wait_limit, abort_flag)) { dead = true; break; }
            tc_fence_after();
            const uint32_t ta = ta0 + sa * (uint32_t)A_COLS;
            const uint64_t bd = bdesc0 + (uint64_t)(((uint32_t)slot * (uint32_t)B_SLOT) >> 4);
            for (slot += NISS; slot >= BS;) slot -= BS;
            // slice s of 16 k is 32 bytes (s % 4) of activation tile s / 4
            if (leader) {
#pragma unroll
                for (int j = 0; j < STEP_TILES * 4; j++) {
                    const uint64_t bj = bd + (uint64_t)(((uint32_t)((j >> 2) * B_TILE) + (uint32_t)((j & 3) * 32)) >> 4);
                    umma_f16_ta(acc, ta + (uint32_t)(8 * j), bj, idesc, (i > iw || j > 0) ? 1u : 0u);
                    if (FMT == FMT_Q4_0) umma_f16_ta(acc, ta + (uint32_t)(32 + 8 * j), bj, idesc, 1u);
                }
                umma_commit(smem_u32(&step_done[i % NBAR]));
            }
            __syncwarp();
        }
        if (!dead && n_steps > iw) {   // drain: this warp's last step
            const int last = iw + (n_steps - 1 - iw) / NISS * NISS;
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
    float *red = reinterpret_cast<float *>(b_s);   // [NB cols][128 rows]
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
                for (int j = 0; j < 16; j++) v[j] = __uint_as_float(a0[j]) + (n_steps > 1 ? __uint_as_float(a1[j]) : 0.f);   // (one step: one accumulator)
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 16; j++) red[(c0 + j) * ROWS + lrow] = v[j];
        }
    }
    const int cols = min(p.NB, p.m - m0), r4 = lane * 4;
    auto store_rows = [&](int col, float4 a) {   // a warp finishes a column: 32 x 4 rows
        OutT *dst = out + (size_t)(m0 + col) * n_rows + n0 + r4;
        if (n0 + r4 + 3 < n_rows && (((uintptr_t)dst) & (4 * sizeof(OutT) - 1)) == 0) {
            store_c4(dst, a);
        } else {
            const float e[4] = {a.x, a.y, a.z, a.w};
            for (int q = 0; q < 4; q++)
                if (n0 + r4 + q < n_rows) store_c(dst + q, e[q]);
        }
    };
    if (p.ks > 1) {
        // The ks CTAs of this tile are one cluster; CTA `rank` finishes every ks-th column: adds the partials in split order and stores.
        cluster_sync();
        const int rank = (int)blockIdx.z;
        const uint32_t red_a = smem_u32(red);
        if (!failed) {
            for (int col = rank + p.ks * warp; col < cols; col += p.ks * (NT / 32)) {
                const uint32_t la = red_a + (uint32_t)((col * ROWS + r4) * 4);
                float4 pv[MAX_KS];
#pragma unroll
                for (int sp = 0; sp < MAX_KS; sp++) pv[sp] = sp < p.ks ? ld_dsmem_f4(la, (uint32_t)sp) : make_float4(0.f, 0.f, 0.f, 0.f);
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int sp = 0; sp < MAX_KS; sp++) {
                    a.x += pv[sp].x; a.y += pv[sp].y; a.z += pv[sp].z; a.w += pv[sp].w;
                }
                store_rows(col, a);
            }
        }
        cluster_sync();   // no CTA leaves while a peer may still read its shared memory
    } else {
        // (through shared memory: stored straight from tensor memory, 64 bytes a warp, a 96-column tile took 3500 cycles)
        __syncthreads();
        if (!failed)
            for (int col = warp; col < cols; col += NT / 32) store_rows(col, *reinterpret_cast<const float4 *>(red + col * ROWS + r4));
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

// Batch rows per CTA and K splits of a launch of `tiles` 128-row tiles, the cheapest by an estimate in cycles.  Q4_0: fitted to all plans of 93
// shapes (17 .. 512 rows, K 64 .. 8192, n 128 .. 16384), one call after the other and side by side, where plans of few CTAs win; a split costs by
// its clusters and, in a launch of one wave, by how many CTAs they are.  The plan it picks takes 1.4 % longer than the best one in the mean, 13 % at most (3.5 and 31 % without
// that term: 34 x 512 x 7872 6.9 us in 62 pairs, 5.4 in 62 CTAs; 291 x 512 x 1088 7.0 and 5.5).  TQ2_0 keeps the fit of its own 113 shapes, 2.0 % above the
// best plan: other splits round differently, and in a decode step that flips KV codes.  Clusters cannot use every SM, other launches can.
struct TclPlan {
    int m_tiles, NB, ks, ups, units;   // ks splits of ups units of two steps
    uint64_t waves;
};
static TclPlan tcl_plan(int fmt, const lc_kernels *k, uint32_t m, uint32_t kk, int tiles) {
    const int step_k = fmt == FMT_Q4_0 ? TclFmt<FMT_Q4_0>::step_k : TclFmt<FMT_TQ2_0>::step_k;
    TclPlan pl = {1, 16, 1, 1, ((int)kk + 2 * step_k - 1) / (2 * step_k), 1};
    uint64_t best = ~0ull;
    for (int mt = ((int)m + MAX_NB - 1) / MAX_NB; mt <= ((int)m + 47) / 48; mt++) {
        const int nb = (((int)m + mt - 1) / mt + 15) / 16 * 16, real_mt = ((int)m + nb - 1) / nb;
        for (int ks = 1; ks <= MAX_KS && (ks == 1 || 2 * ks <= pl.units); ks++) {
            const uint64_t at_once = ks > 1 ? k->cluster_cap[ks] : (uint64_t)k->ctx->sm_count, waves = ((uint64_t)tiles * real_mt + at_once - 1) / at_once;
            const uint64_t unit = 910u + (fmt == FMT_Q4_0 ? 4u : 7u) * (uint64_t)nb, ctas = (uint64_t)tiles * real_mt;
            const uint64_t split = ks == 1 ? 0u : fmt == FMT_Q4_0 && waves == 1 ? 800u + (400u + 25u * ctas) * (uint64_t)ks : 2000u + 100u * (uint64_t)ks;
            const uint64_t cost = waves * (6900u + (uint64_t)((pl.units + ks - 1) / ks) * unit + 9u * (uint64_t)nb + split);
            if (cost < best) {
                best = cost;
                pl.m_tiles = real_mt;
                pl.NB = nb;
                pl.ks = ks;
                pl.waves = waves;
            }
        }
    }
    pl.ups = (pl.units + pl.ks - 1) / pl.ks;
    pl.ks = (pl.units + pl.ups - 1) / pl.ups;
    return pl;
}

// What a launch over one Q4_0 matrix takes at 17 .. 64 rows, in ns, for the choice between this kernel and the register-direct one
// (qmatmul_mma.cu) where there are more tiles than SMs; 0 with fewer, where this one is never the slower by more than 1 % (20 x 512 x 6144:
// 5.45 us against 5.41; 24 x 16384 x 256 5.1 / 5.8; 24 x 4096 x 6144 15.4 / 17.4; eight of 24 x 1536 x 512 in one batch 25.8 / 37.7).
// A wave costs its start, 550 a unit of 128 k and 12 a batch column.  Fitted, with the other kernel's estimate, to both kernels' times over 1900 shapes
// (n 19000 .. 262144, K 64 .. 1536, 17 .. 64 rows): the kernel that it picks takes 0.3 % longer than the faster one in the mean, more than 5 % at 2 % of
// the shapes, 18 % at most (64 x 64 x 44000).  Among those that an older fit gave to the other kernel: 24 x 512 x 32000 13.0 us there, 10.2 here; 24 x 896 x
// 44000 25.0 / 19.5; 24 x 768 x 262144 94.1 / 89.7.
uint64_t lc_qgemm_tcl_estimate(const lc_kernels *k, uint32_t m, uint32_t kk, uint32_t n) {
    const uint64_t tiles = (n + ROWS - 1) / ROWS, sms = (uint64_t)k->ctx->sm_count;
    if (tiles <= sms) return 0;
    const TclPlan pl = tcl_plan(FMT_Q4_0, k, m, kk, (int)tiles);
    return pl.waves * (2300 + 550 * (uint64_t)pl.ups + 12 * (uint64_t)pl.NB);
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
    p.steps = ((int)kk + step_k - 1) / step_k;
    p.m_tiles = pl.m_tiles;
    p.NB = pl.NB;
    p.ks = pl.ks;
    p.sps = 2 * pl.ups;
    if (p.m_tiles > 65535) return -1;
    p.status = k->dev_status;
    p.wait_limit = k->test_wait_expiry ? 4096u : WAIT_LIMIT;
    p.extra_arrivals = k->test_wait_expiry ? 1u : 0u;
    const size_t b_slot = (size_t)(step_k / KT) * p.NB * KT * 2, fixed = (size_t)RAW_SLOTS * RAW_SLOT + 256 + 1024;
    p.b_slots = (int)((220 * 1024 - fixed) / b_slot);
    if (p.b_slots > NBAR) p.b_slots = NBAR;
    if (p.b_slots > p.sps) p.b_slots = p.sps;
    size_t b_bytes = b_slot * p.b_slots;
    if (b_bytes < (size_t)ROWS * p.NB * 4) b_bytes = (size_t)ROWS * p.NB * 4;
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
