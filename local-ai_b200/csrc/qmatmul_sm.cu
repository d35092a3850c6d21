// Small-batch quantized matmul C[m, n] = A[m, K] (f16) x W[n, K]^T, W in GGUF Q4_0 / TQ2_0 blocks, m <= 16: the projections
// of one token or of a small decode batch (shaders/matvec_quant.metal:64-387 and the m <= 8 kernels at :389-577), alone, up
// to three matrices on the same activations, or gate and up of a GeGLU pair (local-engine/src/layer.rs:825-838).
//
// Such a projection is a few megabytes that sit behind the kernel before it, so what counts is the chain after that kernel
// has finished: read the activations, multiply, add up, store.  The chain here has no shared-memory staging of the
// activations, no tensor memory and no exchange between CTAs:
//   * a CTA owns 16 / 32 / 64 weight rows and all of K; its raw blocks come in by bulk copy (COPY_ROWS .. below) before the
//     dependency wait, and the CTA is small enough that the next launch's CTAs become resident and fetch theirs meanwhile;
//   * the twelve warps split K into 128-k steps: a warp reads its part of the activations straight into MMA fragments,
//     16 bytes per lane, all of them in flight together; K is permuted so that a lane's weights come from the code bytes it
//     holds and its activations are contiguous;
//   * the warps' partial sums meet once in shared memory and are added in a fixed order.
// Issue slots bound what is left, so the conversion of the weights is two instructions per two of them: codes masked in place
// are f16 subnormals, q 4^l 2^-24 (TQ2_0, bit pair l of a byte) or q 16^l 2^-24 (Q4_0, nibble l), and one multiply-add makes
// them (q - z) 2^-9, exactly and at one scale.  The operands are integers times a power of two; every block's sum is scaled by
// d 2^9 in f32, the reference's d * sum((q - z) x).  (With a byte table and permutes, as the tcgen05 kernels decode, the
// kernel issued twice the instructions and 8192 x 1536 at m = 1 took 6.1 us.  Leaving z to a sum of the activations saves
// the multiply-add but cancels: twice the rounding error.)
#include <stdlib.h>

#include "lc_internal.h"
#include "qm_codes.cuh"
#include "tensor_map.h"

namespace {

constexpr int FMT_Q4_0 = 0, FMT_TQ2_0 = 1;
constexpr int SM_NW = 12, SM_NT = SM_NW * 32, SM_UNIT = 128;   // warps (each a part of K), threads, k per step of a warp
constexpr int SM_GROUPS = 3;
constexpr uint32_t SM_WAIT_LIMIT = 1u << 22;
// A bulk copy takes the copy engine some 70 cycles however short it is, and a CTA has up to 64 rows: rows below 2 KB come in together, as the
// one range that they are, or, where rows a multiple of 64 bytes long would start in the same few banks, as a box of a tensor map
// 16 bytes wider than the matrix.  (35 matrices in a graph, side by side, against a copy per row: TQ2_0 8192 x 1536 at one row 84.0 -> 65.6 us, at
// 16 rows 101.0 -> 84.2; Q4_0 6144 x 1536 at one row 115 -> 102.  Enqueued call by call the host sets the pace, 2.6 to 3.1 us a call
// from box to box, and 16 rows take 95 to 109 us either way.)  Kernels of their own: decided at run time it cost CTAs of 16 rows 3 %.
constexpr int COPY_ROWS = 0, COPY_RANGE = 1, COPY_BOX = 2;

struct SmParams {
    const uint8_t *w[SM_GROUPS];
    void *out[SM_GROUPS];
    int n[SM_GROUPS], tile_end[SM_GROUPS];
    int ngroups;
    const __half *x;
    int m, K, nb;          // nb = blocks per weight row
    int raw_rs;            // bytes from row to row of raw blocks
    int *status;
    uint32_t wait_limit;
    uint32_t extra_arrivals;   // 0; 1 in the expiry self-test
    uint32_t order;            // LcOrder::flags
};

struct SmBoxParams : SmParams {
    CUtensorMap w_map;
};
template <int COPY> struct SmArg { typedef SmParams type; };
template <> struct SmArg<COPY_BOX> { typedef SmBoxParams type; };

__device__ __forceinline__ void sm_store(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void sm_store(float *p, float v) { *p = v; }
__device__ __forceinline__ void sm_store2(__half *p, float2 v) { *reinterpret_cast<__half2 *>(p) = __floats2half2_rn(v.x, v.y); }
__device__ __forceinline__ void sm_store2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ void sm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// N consecutive 32-bit words at a 2-byte aligned shared-memory address, the bytes of each in the order 0, 2, 1, 3: a mask
// then pairs neighbouring codes in the halves of a register.
template <int N>
__device__ __forceinline__ void lds_codes(uint32_t a, uint32_t (&w)[N]) {
    const uint32_t sel = (a & 2u) ? 0x5342u : 0x3120u, base = a & ~3u;
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; i++) r[i] = lds32(base + 4 * i);
#pragma unroll
    for (int i = 0; i < N; i++) w[i] = __byte_perm(r[i], r[i + 1], sel);
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
    return v;
}

__host__ __device__ __forceinline__ int raw_bytes(int rows, int rs) { return (rows * rs + 15) / 16 * 16; }

// NT8: batch columns / 8.  MTW: 16-row tiles of the CTA (every warp works on all of them).  SINGLE: a warp has at most one
// step, so a tile's sums go to shared memory at once and four tiles fit the registers of two CTAs per SM.
template <int FMT, int NT8, int MTW, bool SINGLE, int COPY, bool GEGLU, typename OutT, bool ORDERED>
__global__ void __launch_bounds__(SM_NT, NT8 == 2 && !SINGLE ? 1 : 2)
qgemm_sm_kernel(const __grid_constant__ typename SmArg<COPY>::type p) {
    constexpr int BB = FMT == FMT_Q4_0 ? 18 : 66;
    constexpr int ROWS = MTW * 16, OROWS = GEGLU ? ROWS / 2 : ROWS;
    constexpr int RS = ROWS + 4;                // padded column of partial sums
    lc_order_begin<ORDERED>(p.order);
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    uint8_t *raw = smem;                                                       // [ROWS][raw_rs]
    float *red = reinterpret_cast<float *>(smem + raw_bytes(ROWS, p.raw_rs));  // [SM_NW][NT8 * 8][RS]
    __shared__ __align__(8) uint64_t raw_full;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    int grp = 0;
    if (!GEGLU)
        while (grp + 1 < p.ngroups && (int)blockIdx.x >= p.tile_end[grp]) grp++;
    const int n0 = ((int)blockIdx.x - (grp ? p.tile_end[grp - 1] : 0)) * OROWS;   // first output row
    const int n_rows = p.n[grp];
    const size_t rb = (size_t)p.nb * BB, w_bytes = rb * (size_t)n_rows;

    // ---- before the dependency wait: the raw blocks (constant operands) ----
    const uint32_t bar = smem_u32(&raw_full);
    if (tid == 0) {
        mbar_init(bar, (COPY == COPY_ROWS ? ROWS : 1) + p.extra_arrivals);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if constexpr (COPY == COPY_BOX) {
            mbar_arrive_expect_tx(bar, (uint32_t)(ROWS * p.raw_rs));
            tma_load_2d(smem_u32(raw), &p.w_map, 0, n0, bar);
        } else if constexpr (COPY == COPY_RANGE) {   // (a tile starts on a multiple of 8 rows of an even number of bytes)
            const uint32_t want = (uint32_t)(min(OROWS, n_rows - n0) * (int)rb);
            const size_t a0 = (size_t)n0 * rb;
            uint32_t bytes = (want + 15u) & ~15u;
            const bool past = a0 + bytes > w_bytes;   // the last bytes of the matrix: nothing is read past its end
            if (past) {
                bytes -= 16;
                for (int h = 0; h < (GEGLU ? 2 : 1); h++)
#pragma unroll 1
                    for (uint32_t i = bytes; i < want; i++) raw[h * OROWS * (int)rb + i] = p.w[GEGLU ? h : grp][a0 + i];
            }
            mbar_arrive_expect_tx(bar, bytes * (GEGLU ? 2u : 1u));
#pragma unroll
            for (int h = 0; h < (GEGLU ? 2 : 1); h++)
                if (bytes) bulk_g2s(smem_u32(raw) + (uint32_t)(h * OROWS * (int)rb), p.w[GEGLU ? h : grp] + a0, bytes, bar);
        }
    }
    __syncthreads();
    if constexpr (COPY == COPY_ROWS) {
        if (tid < ROWS) {
            const int row = n0 + (GEGLU ? tid % OROWS : tid);
            const uint8_t *wm = p.w[GEGLU ? tid / OROWS : grp];
            if (row < n_rows) {
                const size_t g0 = (size_t)row * rb, a0 = g0 & ~(size_t)15;
                uint32_t bytes = (uint32_t)(((g0 + rb - a0) + 15) & ~(size_t)15);
                uint8_t *dst = raw + tid * p.raw_rs;
                if (a0 + bytes > w_bytes) {   // the last bytes of the matrix: nothing is read past its end
                    bytes -= 16;
#pragma unroll 1
                    for (uint32_t i = 0; i < 16; i++) dst[bytes + i] = (a0 + bytes + i < w_bytes) ? wm[a0 + bytes + i] : 0;
                }
                mbar_arrive_expect_tx(bar, bytes);
                if (bytes) bulk_g2s(smem_u32(dst), wm + a0, bytes, bar);
            } else {
                mbar_arrive(bar);
            }
        }
    }
    // this lane's operand rows: 16 mt + g and + 8
    auto row_at = [&](int mt, int h, bool &ok_) -> uint32_t {
        const int r = mt * 16 + h * 8 + g, row = n0 + (GEGLU ? r % OROWS : r);
        ok_ = row < n_rows;
        return smem_u32(raw) + (uint32_t)(r * p.raw_rs) + (COPY == COPY_ROWS ? (uint32_t)(((size_t)row * rb) & 15) : 0u);
    };
    const int units = (p.K + SM_UNIT - 1) / SM_UNIT;
    lc_order_wait<ORDERED>(p.order);

    // ---- activations of one step as B fragments.  TQ2_0: k = 32 l + 8t .. + 7 (l = 0..3), one 16-byte load each.
    //      Q4_0: block l of the step, k = 32 l + 4t .. + 3 and 32 l + 16 + 4t .. + 3, two 8-byte loads. ----
    uint4 xr[NT8][4];
    auto load_x = [&](int u, uint4 (&x)[NT8][4]) {
#pragma unroll
        for (int nt = 0; nt < NT8; nt++) {
            const int col = nt * 8 + g;
            const __half *src = p.x + (size_t)col * p.K + (size_t)u * SM_UNIT;
#pragma unroll
            for (int l = 0; l < 4; l++) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (col < p.m && u < units && (FMT == FMT_TQ2_0 || u * 4 + l < p.nb)) {
                    if (FMT == FMT_TQ2_0) {
                        v = *reinterpret_cast<const uint4 *>(src + 32 * l + 8 * t);
                    } else {
                        const uint2 lo = *reinterpret_cast<const uint2 *>(src + 32 * l + 4 * t), hi = *reinterpret_cast<const uint2 *>(src + 32 * l + 16 + 4 * t);
                        v = make_uint4(lo.x, lo.y, hi.x, hi.y);
                    }
                }
                x[nt][l] = v;
            }
        }
    };
    load_x(warp, xr);
    bool ok;
    {
        uint32_t w = 1;
        if (lane == 0) w = mbar_wait(bar, 0u, p.wait_limit) ? 1u : 0u;
        ok = __shfl_sync(0xffffffffu, w, 0);
    }
    // acc += this step's part of rows 16 mt + g, + 8
    auto step = [&](int u, int mt, const uint4 (&x)[NT8][4], float (&acc)[NT8][4]) {
        bool rok[2];
        const uint32_t ra[2] = {row_at(mt, 0, rok[0]), row_at(mt, 1, rok[1])};
        if constexpr (FMT == FMT_TQ2_0) {
            uint32_t cw[2][2], sh[2][2];
            float d[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t a = ra[h] + (uint32_t)((u >> 1) * BB);
                lds_codes<2>(a + (uint32_t)(32 * (u & 1) + 8 * t), cw[h]);
                sh[h][0] = cw[h][0] >> 8;
                sh[h][1] = cw[h][1] >> 8;
                d[h] = rok[h] ? __half2float(__ushort_as_half((unsigned short)lds16(a + 64u))) * 512.0f : 0.f;
            }
            float c[2][NT8][4] = {};
#pragma unroll
            for (int l = 0; l < 4; l++) {
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const uint32_t a0 = codes_f16<2, 1>(cw[0][q], l), a1 = codes_f16<2, 1>(cw[1][q], l), a2 = codes_f16<2, 1>(sh[0][q], l),
                                   a3 = codes_f16<2, 1>(sh[1][q], l);
#pragma unroll
                    for (int nt = 0; nt < NT8; nt++) sm_mma(c[q][nt], a0, a1, a2, a3, q ? x[nt][l].z : x[nt][l].x, q ? x[nt][l].w : x[nt][l].y);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT8; nt++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[nt][i] = fmaf(c[0][nt][i] + c[1][nt][i], d[i >> 1], acc[nt][i]);
        } else {
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const int blk = u * 4 + l;
                if (blk >= p.nb) break;
                uint32_t cw[2], sh[2];
                float d[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t a = ra[h] + (uint32_t)(blk * BB);
                    uint32_t w[1];
                    lds_codes<1>(a + 2u + (uint32_t)(4 * t), w);
                    cw[h] = w[0];
                    sh[h] = w[0] >> 8;
                    d[h] = rok[h] ? __half2float(__ushort_as_half((unsigned short)lds16(a))) * 512.0f : 0.f;
                }
#pragma unroll
                for (int nt = 0; nt < NT8; nt++) {
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
                    sm_mma(c, codes_f16<4, 8>(cw[0], 0), codes_f16<4, 8>(cw[1], 0), codes_f16<4, 8>(sh[0], 0), codes_f16<4, 8>(sh[1], 0), x[nt][l].x, x[nt][l].y);
                    sm_mma(c, codes_f16<4, 8>(cw[0], 1), codes_f16<4, 8>(cw[1], 1), codes_f16<4, 8>(sh[0], 1), codes_f16<4, 8>(sh[1], 1), x[nt][l].z, x[nt][l].w);
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[nt][i] = fmaf(c[i], d[i >> 1], acc[nt][i]);
                }
            }
        }
    };
    // this warp's sums of a tile into shared memory
    auto put = [&](int mt, const float (&acc)[NT8][4]) {
#pragma unroll
        for (int nt = 0; nt < NT8; nt++)
#pragma unroll
            for (int i = 0; i < 4; i++) red[(warp * (NT8 * 8) + nt * 8 + 2 * t + (i & 1)) * RS + mt * 16 + g + 8 * (i >> 1)] = acc[nt][i];
    };
    if constexpr (SINGLE) {
#pragma unroll 1
        for (int mt = 0; mt < MTW; mt++) {
            float acc[NT8][4];
#pragma unroll
            for (int nt = 0; nt < NT8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            if (ok && warp < units) step(warp, mt, xr, acc);
            put(mt, acc);
        }
    } else {
        float acc[MTW][NT8][4];
#pragma unroll
        for (int mt = 0; mt < MTW; mt++)
#pragma unroll
            for (int nt = 0; nt < NT8; nt++) acc[mt][nt][0] = acc[mt][nt][1] = acc[mt][nt][2] = acc[mt][nt][3] = 0.f;
        if (ok) {
            for (int u = warp; u < units; u += SM_NW) {
                uint4 x[NT8][4];
#pragma unroll
                for (int nt = 0; nt < NT8; nt++)
#pragma unroll
                    for (int l = 0; l < 4; l++) x[nt][l] = xr[nt][l];
                load_x(u + SM_NW, xr);
#pragma unroll
                for (int mt = 0; mt < MTW; mt++) step(u, mt, x, acc[mt]);
            }
        }
#pragma unroll
        for (int mt = 0; mt < MTW; mt++) put(mt, acc[mt]);
    }
    const bool failed = __syncthreads_or(!ok);
    if (failed) {
        tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED_TCD, tid);
        lc_order_end<ORDERED>(p.order);
        return;
    }
    const int parts = min(units, SM_NW);
    auto total = [&](int col, int r) -> float2 {   // rows r, r + 1
        float2 s = make_float2(0.f, 0.f);
        const float *src = red + col * RS + r;
#pragma unroll 4
        for (int i = 0; i < parts; i++) {
            const float2 v = *reinterpret_cast<const float2 *>(src + i * (NT8 * 8) * RS);
            s.x += v.x;
            s.y += v.y;
        }
        return s;
    };
    OutT *out = reinterpret_cast<OutT *>(p.out[grp]);
    const bool pairs = (n_rows & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & (2 * sizeof(OutT) - 1)) == 0;   // (n0 is even)
    for (int i = tid; i < OROWS / 2 * p.m; i += SM_NT) {
        const int r = 2 * (i % (OROWS / 2)), col = i / (OROWS / 2);
        if (n0 + r >= n_rows) continue;
        float2 v = total(col, r);
        if (GEGLU) {
            const float2 up = total(col, r + OROWS);
            v = make_float2(geglu_f(v.x, up.x), geglu_f(v.y, up.y));
        }
        OutT *dst = out + (size_t)col * n_rows + n0 + r;
        if (pairs) {
            sm_store2(dst, v);
        } else {
            sm_store(dst, v.x);
            if (n0 + r + 1 < n_rows) sm_store(dst + 1, v.y);
        }
    }
    lc_order_end<ORDERED>(p.order);
}

template <int FMT, int NT8, int MTW, bool SINGLE, int COPY, bool GEGLU, typename OutT, bool ORDERED>
int launch_sm(lc_batch *b, bool serial, const SmBoxParams &p, int tiles) {
    auto kern = qgemm_sm_kernel<FMT, NT8, MTW, SINGLE, COPY, GEGLU, OutT, ORDERED>;
    const size_t smem = 128 + raw_bytes(MTW * 16, p.raw_rs) + sizeof(float) * SM_NW * NT8 * 8 * (MTW * 16 + 4);
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    LC_LAUNCH_CHECKED(lc_launch_as(serial, kern, dim3(tiles), dim3(SM_NT), smem, b, static_cast<const typename SmArg<COPY>::type &>(p)));
    b->dispatch_count++;
    return LC_OK;
}
// (rows of one step per warp are below 2 KB, TQ2_0's are one range then, and CTAs of 16 rows copy row by row)
template <int FMT, int NT8, int MTW, bool SINGLE, bool GEGLU, typename OutT, bool ORDERED>
int launch_copy(lc_batch *b, bool serial, const SmBoxParams &p, int tiles, int copy) {
    if constexpr (FMT == FMT_Q4_0)
        if (copy == COPY_BOX) return launch_sm<FMT, NT8, MTW, SINGLE, COPY_BOX, GEGLU, OutT, ORDERED>(b, serial, p, tiles);
    if constexpr (!SINGLE || FMT == FMT_Q4_0)
        if (copy == COPY_ROWS) return launch_sm<FMT, NT8, MTW, SINGLE, COPY_ROWS, GEGLU, OutT, ORDERED>(b, serial, p, tiles);
    return launch_sm<FMT, NT8, MTW, SINGLE, COPY_RANGE, GEGLU, OutT, ORDERED>(b, serial, p, tiles);
}
template <int FMT, int NT8, bool GEGLU, typename OutT, bool ORDERED>
int launch_rows(lc_batch *b, bool serial, const SmBoxParams &p, int tiles, int rows, int copy) {
    if (p.K <= SM_NW * SM_UNIT) {
        if (rows == 64) return launch_copy<FMT, NT8, 4, true, GEGLU, OutT, ORDERED>(b, serial, p, tiles, copy);
        if (rows == 32) return launch_copy<FMT, NT8, 2, true, GEGLU, OutT, ORDERED>(b, serial, p, tiles, copy);
        return launch_sm<FMT, NT8, 1, true, COPY_ROWS, GEGLU, OutT, ORDERED>(b, serial, p, tiles);
    }
    if (rows == 32) return launch_copy<FMT, NT8, 2, false, GEGLU, OutT, ORDERED>(b, serial, p, tiles, copy);
    return launch_sm<FMT, NT8, 1, false, COPY_ROWS, GEGLU, OutT, ORDERED>(b, serial, p, tiles);
}
template <int FMT, bool GEGLU, typename OutT>
int launch_nt(lc_batch *b, bool serial, const SmBoxParams &p, int tiles, int rows, int copy) {
    if (p.order)
        return p.m <= 8 ? launch_rows<FMT, 1, GEGLU, OutT, true>(b, serial, p, tiles, rows, copy) : launch_rows<FMT, 2, GEGLU, OutT, true>(b, serial, p, tiles, rows, copy);
    return p.m <= 8 ? launch_rows<FMT, 1, GEGLU, OutT, false>(b, serial, p, tiles, rows, copy) : launch_rows<FMT, 2, GEGLU, OutT, false>(b, serial, p, tiles, rows, copy);
}

}  // namespace

// Grouped launch: `ng` matrices [ns[g], kk] on the same activations `input` [m, kk]; with `geglu` (TQ2_0), two matrices of one
// shape and one output gelu_tanh(x Wg^T) * (x Wu^T).  Returns LC_OK after a launch, a positive status on error, or -1 when
// the shape is outside what this kernel covers.
int lc_qgemm_sm_launch(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                       lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk, bool geglu) {
    if (m < 1 || m > 16 || ng < 1 || ng > SM_GROUPS || !lc_aligned(input->dptr, 16)) return -1;
    if (geglu && (ng != 2 || ns[0] != ns[1] || fmt != FMT_TQ2_0 || f32out)) return -1;
    if (fmt == FMT_Q4_0 && kk % 4 != 0) return -1;
    SmBoxParams p;
    p.x = (const __half *)input->dptr;
    p.m = (int)m;
    p.K = (int)kk;
    p.nb = (int)(fmt == FMT_Q4_0 ? kk / 32 : kk / 256);
    p.ngroups = geglu ? 1 : ng;
    const size_t rb = (size_t)p.nb * (fmt == FMT_Q4_0 ? 18 : 66);
    // a row's enclosing 16-byte range; an odd number of 32-byte pieces spreads the lanes' rows over the banks
    size_t rs = (rb + 15 + 15) / 16 * 16;
    rs += (32 + 64 - rs % 64) % 64;
    uint64_t rows_all = 0;
    for (int g = 0; g < ng; g++) rows_all += ns[g];
    // Rows per CTA: the fewest CTAs that still give every SM one (a CTA reads all activations), but never so many rows that
    // the raw blocks of two CTAs do not fit an SM together (the next launch's CTA fetches its blocks while this one runs).
    const size_t room = 100 * 1024, sms = (size_t)k->ctx->sm_count;
    int rows = kk <= SM_NW * SM_UNIT ? 64 : 32;
    while (rows > 16 && ((rows_all + rows - 1) / rows < sms * 3 / 4 || rows * rs > room)) rows >>= 1;
    // ... and, where registers leave an SM one CTA (more than 8 batch rows, several steps per warp), not a little over one wave.
    if (rows == 16 && m > 8 && kk > SM_NW * SM_UNIT && (rows_all + 15) / 16 > sms && 32 * rs <= 190 * 1024) rows = 32;
    if (rows * rs > (rows == 32 ? 190 * 1024 : room)) return -1;
    // Q4_0 with few steps per warp, 9 to 16 rows of activations and more than two waves of tiles: the register-direct kernel's
    // 64-row tiles read the activations half as often (11 x 1792 x 15996: 18.0 us here, 13.7 there, 16 x 2048 x 12000 15.0 and 12.9; at K = 3072 24 against 28).
    if (fmt == FMT_Q4_0 && !f32out && m > 8 && kk > SM_NW * SM_UNIT && kk <= 2560 && (rows_all + 31) / 32 > 2 * sms) return -1;
    // A box costs the host 0.1 us a launch, which shows where launches side by side keep up with it (35 of 4000 x 2048 at three rows 93 us with a
    // copy per row, 99 with boxes).
    // (CTAs of 16 rows keep a copy per row: 1024 x 1024 Q4_0 at one row 1.62 us against 1.64 for a box, 1024 x 512 1.49 / 1.54 for a range.)
    int copy = COPY_ROWS;
    if (rb < 2048 && rows >= 32) {
        if (fmt != FMT_Q4_0 || rb % 64 != 0) copy = COPY_RANGE;
        else if (ng == 1 && rows_all * kk >= 1u << 24) copy = COPY_BOX;
    }
    int tiles = 0;
    const int orows = geglu ? rows / 2 : rows;
    for (int g = 0; g < SM_GROUPS; g++) {
        const int gi = g < ng ? g : ng - 1;
        if (!lc_aligned(weights[gi]->dptr, 16)) return -1;
        p.w[g] = (const uint8_t *)weights[gi]->dptr;
        p.out[g] = outputs[gi]->dptr;
        p.n[g] = (int)ns[gi];
        if (g < ng && !(geglu && g > 0)) tiles += ((int)ns[g] + orows - 1) / orows;
        p.tile_end[g] = tiles;
    }
    if (tiles < 1) return -1;
    if (copy == COPY_BOX && !lc_wider_rows_map(&p.w_map, k->test_map_refused, p.w[0], rb, ns[0], (uint32_t)rows)) copy = COPY_ROWS;
    p.raw_rs = (int)(copy == COPY_RANGE ? rb : copy == COPY_BOX ? rb + 16 : rs);
    p.status = k->dev_status;
    p.wait_limit = k->test_wait_expiry ? 4096u : SM_WAIT_LIMIT;
    p.extra_arrivals = k->test_wait_expiry ? 1u : 0u;
    size_t w_bytes[SM_GROUPS], out_bytes[SM_GROUPS];
    for (int g = 0; g < ng; g++) {
        w_bytes[g] = rb * ns[g];
        out_bytes[g] = (size_t)m * ns[g] * (f32out ? 4 : 2);
    }
    // Weights up to which 35 such launches one after the other keep up with the host (2.5 us each).  On the lines' two sides, side by side against
    // that: Q4_0, 2.1 M 1.02 / 3.1 M 0.77 at up to four rows, 1.6 M 1.02 / 2.1 M 0.79 at eight, 0.5 M 0.89 at sixteen; TQ2_0, 3.1 M 1.02 / 4.2 M 0.94 at up to
    // eight, 1.6 M 1.04 / 2.1 M 0.98 at sixteen.
    const size_t host_paced = fmt == FMT_Q4_0 ? (m <= 4 ? 5u << 19 : m <= 8 ? 7u << 18 : 3u << 17) : (m <= 8 ? 7u << 19 : 7u << 18);
    size_t n_all = 0;
    for (int g = 0; g < ng; g++) n_all += ns[g];
    LcOrder order(b, input, (size_t)m * kk * 2, ng, weights, w_bytes, outputs, out_bytes, n_all * kk <= host_paced);
    p.order = order.flags;
    int st;
    if (geglu) st = launch_nt<FMT_TQ2_0, true, __half>(b, order.serial, p, tiles, rows, copy);
    else if (fmt == FMT_Q4_0) st = f32out ? launch_nt<FMT_Q4_0, false, float>(b, order.serial, p, tiles, rows, copy) : launch_nt<FMT_Q4_0, false, __half>(b, order.serial, p, tiles, rows, copy);
    else st = f32out ? launch_nt<FMT_TQ2_0, false, float>(b, order.serial, p, tiles, rows, copy) : launch_nt<FMT_TQ2_0, false, __half>(b, order.serial, p, tiles, rows, copy);
    order.launched = st == LC_OK;
    return st;
}
