// Streaming tensor-core matvec / small-batch matmul (m <= 8) over GGUF Q4_0 / TQ2_0 rows:
//   out[m, n] = X[m, K] (f16) x W[n, K]^T.
// Stands in for matvec_q4_0 / matvec_tq2_0 (+ f32out) and the batchm / smallm kernels of
// shaders/matvec_quant.metal (:64-312, :590-916) when the matrix is large enough for bandwidth to matter.
//
// A batch-1 matvec is HBM-bound in principle, but on CUDA cores the dequantisation costs 5-6 instructions per
// weight and binds long before HBM does.  Here the multiply-adds run on mma.sync (the 1..8 batch rows take the
// MMA's N = 8), which leaves about two integer instructions per four weights:
//   * a persistent CTA streams groups of 64 consecutive weight rows -- one contiguous byte range, so a group is one bulk
//     copy and DRAM sees sequential reads -- through a ring of three slots; a warp of its own fetches, and the others
//     meet it at mbarriers only, so a warp that is done with a group goes on to the next;
//   * the activations (8 rows x K) stay in shared memory, or in registers, for the whole launch;
//   * warp (rg, kq) of 16 owns rows 16 rg .. + 15 of the group and quarter kq of K; its threads turn 2-byte pieces
//     of code bytes into A fragments in registers (thread t of a quad owns bytes 2t, 2t+1 of every 8-byte group);
//   * the four K quarters meet at a barrier of their four warps, and each adds and stores a quarter of the sums.
// Numerics keep the exact-weight semantic of the CUDA-core kernels: the A operand holds the integers q - z (times 2^-9), every
// block (Q4_0) or half block (TQ2_0) is accumulated on its own and scaled by d in f32.  Accumulation is f32.
// Issue slots bound it: 2-byte shared loads, masks, one multiply-add per two weights.  262144 x 1536 Q4_0 at m = 1 takes 57.4 us
// (3.95 TB/s); 67 us with cp.async by every thread, two barriers of the whole CTA per group and permutes for the conversion.
// TQ2_0 gains more, as its conversion had a permute and a multiply per two weights: 90 matrices of 8192 x 1536 in one
// launch 2.4 -> 1.6 us each.
#include "lc_internal.h"
#include "qm_codes.cuh"
#include "tcgen05_util.cuh"

namespace {

constexpr int FMT_Q4_0 = 0;
constexpr int FMT_TQ2_0 = 1;
constexpr int NW = 16, NT = (NW + 1) * 32;   // sixteen working warps and one that fetches
constexpr uint32_t STREAM_WAIT_LIMIT = 1u << 22;   // a constant: read from the parameters for the expiry self-test it cost 1 - 2 % (57.7 -> 58.3 .. 59.0 us)
constexpr int GROUP_ROWS = 64;       // rows per ring slot: 4 row groups of 16
constexpr int SLOTS = 3;
constexpr int UNIT_K = 128;          // K is split over the four warp quarters in units of 128 k

constexpr int MAX_MATRICES = 96;     // matrices of one shape streamed by one launch (lc_matvec_*_group_into)

struct StreamParams {
    const uint8_t *w[MAX_MATRICES];   // n_mat matrices of n rows each, all read against the same activations
    void *out[MAX_MATRICES];
    const __half *x;
    int n, m, K, nb;        // nb = blocks per row
    int gpm;                // 64-row groups per matrix: ceil(n / 64)
    int groups;             // n_mat * gpm
    int xs;                 // bytes per activation row in shared memory
    int slot_bytes;         // bytes reserved per ring slot
    int *status;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes = 16u) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x2(uint32_t &b0, uint32_t &b1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];\n" : "=r"(b0), "=r"(b1) : "r"(addr));
}
__device__ __forceinline__ void store_c(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store_c(float *p, float v) { *p = v; }
__device__ __forceinline__ uint32_t lds_u16(const uint8_t *p) { return *reinterpret_cast<const uint16_t *>(p); }

template <int FMT> struct Fmt;
template <> struct Fmt<FMT_Q4_0> { static constexpr int bytes = 18; };
template <> struct Fmt<FMT_TQ2_0> { static constexpr int bytes = 66; };

// UPQ > 0: the warp's K quarter is UPQ units long and its activation fragments (8 k-steps x 2 registers per unit)
// stay in registers for the whole launch; UPQ = 0: any length, fragments re-read from shared memory with ldmatrix.
// MULTI: several matrices (group index -> matrix and group of it); otherwise the one matrix p.w[0].
template <int FMT, typename OutT, int UPQ, bool MULTI>
__global__ void __launch_bounds__(NT, 1) qgemv_mma_stream_kernel(const __grid_constant__ StreamParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int BB = Fmt<FMT>::bytes;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int rg = warp & 3, kq = warp >> 2;
    lc_pdl_trigger();
    const size_t rb = (size_t)p.nb * BB, w_bytes = rb * (size_t)p.n;
    uint8_t *x_s = smem;                                              // [8][xs]
    float4 *red = reinterpret_cast<float4 *>(smem + 8 * p.xs);        // [2][NW][32]
    uint8_t *ring = smem + 8 * p.xs + 2 * NW * 32 * 16;               // [SLOTS][slot_bytes]
    const int my_groups = (p.groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    __shared__ __align__(8) uint64_t full_s[SLOTS], empty_s[SLOTS];
    __shared__ int abort_s;
    volatile int *abort_flag = &abort_s;
    const uint32_t full = smem_u32(full_s), empty = smem_u32(empty_s);
    // Group `it` of this CTA: group (blockIdx.x + it gridDim.x) of the launch = rows 64 gi .. of matrix mi; one contiguous byte
    // range, one bulk copy (one thread).
    auto load_group = [&](int it) {
        const int gl = (int)blockIdx.x + it * (int)gridDim.x, mi = MULTI ? gl / p.gpm : 0, grp = gl - mi * p.gpm;
        const uint8_t *wm = p.w[mi];
        const size_t start = (size_t)grp * GROUP_ROWS * rb;
        const size_t len = (size_t)min(GROUP_ROWS, p.n - grp * GROUP_ROWS) * rb;
        const size_t a0 = start & ~(size_t)15;
        uint32_t bytes = (uint32_t)((start - a0 + len + 15) & ~(size_t)15);
        uint8_t *slot = ring + (size_t)(it % SLOTS) * p.slot_bytes;
        if (a0 + bytes > w_bytes) {   // nothing is read past the matrix's end
            bytes -= 16;
            for (uint32_t b = 0; b < 16; b++) slot[bytes + b] = (a0 + bytes + b < w_bytes) ? wm[a0 + bytes + b] : 0;
        }
        mbar_arrive_expect_tx(full + 8 * (it % SLOTS), bytes);
        if (bytes) bulk_g2s(smem_u32(slot), wm + a0, bytes, full + 8 * (it % SLOTS));
    };
    // the weights of the first groups do not depend on the previous kernel
    if (tid == NW * 32) {
        for (int s = 0; s < SLOTS; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, NW);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int it = 0; it < SLOTS && it < my_groups; it++) load_group(it);
    }
    lc_pdl_wait();
    for (int i = tid; i < 8 * (p.K / 8); i += NT) {
        const int r = i / (p.K / 8), pc = i - r * (p.K / 8);
        const bool ok = r < p.m;
        cp_async16(smem_u32(x_s + r * p.xs + pc * 16), ok ? (const void *)(p.x + (size_t)r * p.K + pc * 8) : (const void *)p.x,
                   ok ? 16u : 0u);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();          // the activations have landed, the barriers are ready
    bool alive = true;   // no wait of this warp has run out
    auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool {
        if (alive && !mbar_wait_warp(bar, parity, STREAM_WAIT_LIMIT)) {
            alive = false;
            *abort_flag = 1;
        }
        return alive;
    };
    if (warp == NW) {
        for (int it = SLOTS; it < my_groups; it++) {
            if (!warp_wait(empty + 8 * (it % SLOTS), (uint32_t)((it / SLOTS - 1) & 1))) break;
            if (lane == 0) load_group(it);
            __syncwarp();
        }
    } else {
    // this warp's quarter of K, in units of 128 k
    const int nu = p.K / UNIT_K, upq = (nu + 3) / 4;
    const int u0 = kq * upq, u1 = min(nu, u0 + upq);
    // ldmatrix.x2 lane address: lanes 0-7 rows of the first k half, lanes 8-15 the second
    const uint32_t xl = smem_u32(x_s) + (uint32_t)((lane & 7) * p.xs + ((lane >> 3) & 1) * 16);
    uint32_t breg[UPQ > 0 ? UPQ * 8 : 1][2];
    // Code bytes 2t, 2t + 8 pair up in a register, and so do 2t + 1, 2t + 9: the activations' k follow.
    auto load_b = [&](uint32_t &b0, uint32_t &b1, uint32_t addr) {
        uint32_t r0, r1;
        ldmatrix_x2(r0, r1, addr);
        b0 = __byte_perm(r0, r1, 0x5410);
        b1 = __byte_perm(r0, r1, 0x7632);
    };
    if (UPQ > 0) {
#pragma unroll
        for (int uu = 0; uu < (UPQ > 0 ? UPQ : 1); uu++)
#pragma unroll
            for (int s8 = 0; s8 < 8; s8++) {
                breg[uu * 8 + s8][0] = breg[uu * 8 + s8][1] = 0u;
                if (u0 + uu < u1) load_b(breg[uu * 8 + s8][0], breg[uu * 8 + s8][1], xl + (uint32_t)(((u0 + uu) * UNIT_K + 16 * s8) * 2));
            }
    }

    // The four quarters of a group of sixteen rows meet at a named barrier; warp kq adds fragment element kq and stores.
    auto reduce_store = [&](int it) {
        const int gl = (int)blockIdx.x + it * (int)gridDim.x, mi = MULTI ? gl / p.gpm : 0, grp = gl - mi * p.gpm;
        const float *rp = reinterpret_cast<const float *>(red + (size_t)(it & 1) * NW * 32 + rg * 32 + lane) + kq;
        const float v = ((rp[0] + rp[4 * 32 * 4]) + rp[2 * 4 * 32 * 4]) + rp[3 * 4 * 32 * 4];
        const int row = grp * GROUP_ROWS + rg * 16 + g + 8 * (kq >> 1), col = 2 * t + (kq & 1);
        if (row < p.n && col < p.m) store_c(reinterpret_cast<OutT *>(p.out[mi]) + (size_t)col * p.n + row, v);
    };

    for (int it = 0; it < my_groups; it++) {
        // (an expired wait does not leave the loop: the other quarters count on this warp at their barrier)
        const bool landed = warp_wait(full + 8 * (it % SLOTS), (uint32_t)((it / SLOTS) & 1));
        const int gl = (int)blockIdx.x + it * (int)gridDim.x, grp = MULTI ? gl % p.gpm : gl;
        const size_t start = (size_t)grp * GROUP_ROWS * rb;
        const uint8_t *slot = ring + (size_t)(it % SLOTS) * p.slot_bytes + (start & 15);
        const uint8_t *rbase[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = rg * 16 + g + 8 * i;
            rbase[i] = slot + (size_t)r * rb;   // (rows past the matrix's last hold leftovers; nothing of them is stored)
        }
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        if (!landed) {
        } else if (FMT == FMT_TQ2_0) {
            // unit u = half h of block b: element 128 h + 32 l + j of the block is bit pair l of code byte 32 h + j
#pragma unroll
            for (int uu = 0; uu < (UPQ > 0 ? UPQ : 64); uu++) {
                const int u = u0 + uu;
                if (u >= u1) break;
                const int b = u >> 1, h = u & 1;
                uint32_t wq[2][2], sh[2][2];
                float df[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint8_t *bp = rbase[i] + b * BB;
                    df[i] = __half2float(*reinterpret_cast<const __half *>(bp + 64)) * 512.0f;
                    const uint8_t *hp = bp + h * 32 + 2 * t;
                    wq[i][0] = lds_u16(hp) | (lds_u16(hp + 8) << 16);
                    wq[i][1] = lds_u16(hp + 16) | (lds_u16(hp + 24) << 16);
                    sh[i][0] = wq[i][0] >> 8;
                    sh[i][1] = wq[i][1] >> 8;
                }
                float cu[2][4] = {};
#pragma unroll
                for (int l = 0; l < 4; l++) {
#pragma unroll
                    for (int qp = 0; qp < 2; qp++) {
                        const uint32_t a[4] = {codes_f16<2, 1>(wq[0][qp], l), codes_f16<2, 1>(wq[1][qp], l), codes_f16<2, 1>(sh[0][qp], l),
                                               codes_f16<2, 1>(sh[1][qp], l)};
                        uint32_t b0, b1;
                        if (UPQ > 0) {
                            b0 = breg[uu * 8 + 2 * l + qp][0];
                            b1 = breg[uu * 8 + 2 * l + qp][1];
                        } else {
                            load_b(b0, b1, xl + (uint32_t)((u * UNIT_K + 32 * l + 16 * qp) * 2));
                        }
                        mma16816(cu[qp], a, b0, b1);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; e++) c[e] = fmaf(df[e >> 1], cu[0][e] + cu[1][e], c[e]);
            }
        } else {
            // unit u = blocks 4u .. 4u+3; block: f16 scale, then byte i holds k = i (low nibble) and i + 16 (high)
#pragma unroll
            for (int uu = 0; uu < (UPQ > 0 ? UPQ : 64); uu++) {
                const int u = u0 + uu;
                if (u >= u1) break;
#pragma unroll
                for (int bi = 0; bi < 4; bi++) {
                    const int b = 4 * u + bi;
                    float df[2];
                    uint32_t wq[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const uint8_t *bp = rbase[i] + b * BB;
                        df[i] = __half2float(*reinterpret_cast<const __half *>(bp)) * 512.0f;
                        wq[i] = lds_u16(bp + 2 + 2 * t) | (lds_u16(bp + 10 + 2 * t) << 16);
                    }
                    float cb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int part = 0; part < 2; part++) {
                        const uint32_t a[4] = {codes_f16<4, 8>(wq[0], part), codes_f16<4, 8>(wq[1], part), codes_f16<4, 8>(wq[0] >> 8, part),
                                               codes_f16<4, 8>(wq[1] >> 8, part)};
                        uint32_t b0, b1;
                        if (UPQ > 0) {
                            b0 = breg[uu * 8 + 2 * bi + part][0];
                            b1 = breg[uu * 8 + 2 * bi + part][1];
                        } else {
                            load_b(b0, b1, xl + (uint32_t)((b * 32 + 16 * part) * 2));
                        }
                        mma16816(cb, a, b0, b1);
                    }
                    c[0] = fmaf(df[0], cb[0], c[0]);
                    c[1] = fmaf(df[0], cb[1], c[1]);
                    c[2] = fmaf(df[1], cb[2], c[2]);
                    c[3] = fmaf(df[1], cb[3], c[3]);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * (it % SLOTS));
        red[((size_t)(it & 1) * NW + kq * 4 + rg) * 32 + lane] = make_float4(c[0], c[1], c[2], c[3]);
        asm volatile("bar.sync %0, 128;\n" ::"r"(1 + rg) : "memory");
        if (landed) reduce_store(it);
    }
    }
    __syncthreads();
    if (*abort_flag) tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, tid);
}

template <int FMT, typename OutT, int UPQ, bool MULTI>
int launch_stream_um(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    auto kern = qgemv_mma_stream_kernel<FMT, OutT, UPQ, MULTI>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    const int grid = p.groups < k->ctx->sm_count ? p.groups : k->ctx->sm_count;
    LC_LAUNCH_CHECKED(lc_launch(kern, dim3(grid), dim3(NT), smem, b, p));
    b->dispatch_count++;
    return LC_OK;
}
template <int FMT, typename OutT, int UPQ>
int launch_stream_u(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    return p.groups > p.gpm ? launch_stream_um<FMT, OutT, UPQ, true>(k, b, p, smem)
                            : launch_stream_um<FMT, OutT, UPQ, false>(k, b, p, smem);
}

template <int FMT, typename OutT>
int launch_stream(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    const int upq = (p.K / UNIT_K + 3) / 4;
    switch (upq) {
        case 1: return launch_stream_u<FMT, OutT, 1>(k, b, p, smem);
        case 2: return launch_stream_u<FMT, OutT, 2>(k, b, p, smem);
        case 3: return launch_stream_u<FMT, OutT, 3>(k, b, p, smem);
        default: return launch_stream_u<FMT, OutT, 0>(k, b, p, smem);
    }
}

}  // namespace

// m <= 8; `count` matrices of one shape [n, kk] against the same activations, each with its own output.  Returns
// LC_OK after a launch, a positive status on error, or -1 when the shape is outside what this kernel covers or too
// small for it to pay (the caller then uses the CUDA-core kernel).
int lc_qgemv_mma_stream_group(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int count,
                              const lc_buf *const *weights, lc_buf *const *outputs, uint32_t m, uint32_t kk, uint32_t n) {
    const int be = fmt == FMT_Q4_0 ? 32 : 256, bb = fmt == FMT_Q4_0 ? 18 : 66;
    if (count < 1 || count > MAX_MATRICES || m > 8 || kk % UNIT_K != 0 || kk % be != 0 || !lc_aligned(input->dptr, 16)) return -1;
    StreamParams p;
    for (int i = 0; i < MAX_MATRICES; i++) {
        const int j = i < count ? i : count - 1;
        if (!lc_aligned(weights[j]->dptr, 16)) return -1;
        p.w[i] = (const uint8_t *)weights[j]->dptr;
        p.out[i] = outputs[j]->dptr;
    }
    p.x = (const __half *)input->dptr;
    p.n = (int)n;
    p.m = (int)m;
    p.K = (int)kk;
    p.nb = (int)(kk / be);
    p.gpm = (int)((n + GROUP_ROWS - 1) / GROUP_ROWS);
    p.status = k->dev_status;
    p.groups = p.gpm * count;
    p.xs = (int)kk * 2 + 16;
    const size_t rb = (size_t)p.nb * bb;
    p.slot_bytes = (int)(((size_t)GROUP_ROWS * rb + 15 + 15) / 16 * 16 + 16);
    const size_t smem = (size_t)8 * p.xs + 2 * NW * 32 * 16 + (size_t)SLOTS * p.slot_bytes;
    if (smem + 256 > k->ctx->smem_optin) return -1;   // (the barriers are static)
    // worth it only when every SM gets a few groups to stream
    if (p.groups < 2 * k->ctx->sm_count) return -1;
    if (fmt == FMT_Q4_0)
        return f32out ? launch_stream<FMT_Q4_0, float>(k, b, p, smem) : launch_stream<FMT_Q4_0, __half>(k, b, p, smem);
    return f32out ? launch_stream<FMT_TQ2_0, float>(k, b, p, smem) : launch_stream<FMT_TQ2_0, __half>(k, b, p, smem);
}

int lc_qgemv_mma_stream(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                        lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    const lc_buf *ws[1] = {weight};
    lc_buf *os[1] = {output};
    return lc_qgemv_mma_stream_group(fmt, f32out, k, b, input, 1, ws, os, m, kk, n);
}
