// Streaming tensor-core matvec / small-batch matmul (m <= 8) over GGUF Q4_0 / TQ2_0 rows:
//   out[m, n] = X[m, K] (f16) x W[n, K]^T.
// Stands in for matvec_q4_0 / matvec_tq2_0 (+ f32out) and the batchm / smallm kernels of
// shaders/matvec_quant.metal (:64-312, :590-916) when the matrix is large enough for bandwidth to matter.
//
// A batch-1 matvec is HBM-bound in principle, but on CUDA cores the dequantisation costs 5-6 instructions per
// weight and binds long before HBM does.  Here the multiply-adds run on mma.sync (the 1..8 batch rows take the
// MMA's N = 8), which leaves about two integer instructions per four weights:
//   * a persistent CTA streams groups of 64 consecutive weight rows -- one contiguous byte range, so a group is one
//     copy and DRAM sees sequential reads -- through a ring of three slots; a warp of its own fetches, and the others
//     meet it at mbarriers only, so a warp that is done with a group goes on to the next;
//   * the activations stay in registers for the whole launch (TQ2_0 rows above 1536: in shared memory);
//   * warp (rg, kq) of 16 owns rows 16 rg .. + 15 of the group and quarter kq of K; its threads turn code bytes into A
//     fragments in registers;
//   * the four K quarters' sums meet in shared memory.
// Numerics keep the exact-weight semantic of the CUDA-core kernels: the A operand holds the integers q - z (times 2^-9), every
// block (Q4_0) or half block (TQ2_0) is accumulated on its own and scaled by d in f32.  Accumulation is f32.
// TQ2_0, 90 matrices of 8192 x 1536 in one launch: 1.6 us each, issue slots (2-byte shared loads, masks, one multiply-add per two
// weights).  Q4_0, 262144 x 1536 at m = 1: 44.7 us (5.1 TB/s), the copies from HBM.
#include "lc_internal.h"
#include "qm_codes.cuh"
#include "tcgen05_util.cuh"
#include "tensor_map.h"

namespace {

constexpr int FMT_Q4_0 = 0;
constexpr int NW = 16, NT = (NW + 1) * 32;   // sixteen working warps and one that fetches
constexpr uint32_t STREAM_WAIT_LIMIT = 1u << 22;   // a constant: read from the parameters for the expiry self-test it cost 1 - 2 % (57.7 -> 58.3 .. 59.0 us)
constexpr int GROUP_ROWS = 64;       // rows per ring slot: 4 row groups of 16
constexpr int SLOTS = 3;             // (Q4_0 rows of 2048 at m > 1 leave room for two)
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
    int pitch, slots;       // Q4_0: bytes from row to row in a slot, ring slots
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
__device__ __forceinline__ float lds_f16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
    return __half2float(__ushort_as_half(v));
}

// Group `it` of this CTA: group (blockIdx.x + it gridDim.x) of the launch = rows 64 gi .. of matrix mi; one contiguous byte
// range, one bulk copy (one thread).
template <bool MULTI>
__device__ __forceinline__ void stream_load(const StreamParams &p, size_t rb, int it, uint8_t *slot, uint32_t full) {
    const int gl = (int)blockIdx.x + it * (int)gridDim.x, mi = MULTI ? gl / p.gpm : 0, grp = gl - mi * p.gpm;
    const uint8_t *wm = p.w[mi];
    const size_t w_bytes = rb * (size_t)p.n, start = (size_t)grp * GROUP_ROWS * rb;
    const size_t len = (size_t)min(GROUP_ROWS, p.n - grp * GROUP_ROWS) * rb;
    const size_t a0 = start & ~(size_t)15;
    uint32_t bytes = (uint32_t)((start - a0 + len + 15) & ~(size_t)15);
    if (a0 + bytes > w_bytes) {   // nothing is read past the matrix's end
        bytes -= 16;
        for (uint32_t b = 0; b < 16; b++) slot[bytes + b] = (a0 + bytes + b < w_bytes) ? wm[a0 + bytes + b] : 0;
    }
    mbar_arrive_expect_tx(full, bytes);
    if (bytes) bulk_g2s(smem_u32(slot), wm + a0, bytes, full);
}

// UPQ > 0: the warp's K quarter is UPQ units long and its activation fragments (8 k-steps x 2 registers per unit)
// stay in registers for the whole launch; UPQ = 0: any length, fragments re-read from shared memory with ldmatrix.
// MULTI: several matrices (group index -> matrix and group of it); otherwise the one matrix p.w[0].
template <typename OutT, int UPQ, bool MULTI>
__global__ void __launch_bounds__(NT, 1) qgemv_tq2_0_stream_kernel(const __grid_constant__ StreamParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int BB = 66;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int rg = warp & 3, kq = warp >> 2;
    lc_pdl_trigger();
    const size_t rb = (size_t)p.nb * BB;
    uint8_t *x_s = smem;                                              // [8][xs]
    float4 *red = reinterpret_cast<float4 *>(smem + 8 * p.xs);        // [2][NW][32]
    uint8_t *ring = smem + 8 * p.xs + 2 * NW * 32 * 16;               // [SLOTS][slot_bytes]
    const int my_groups = (p.groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    __shared__ __align__(8) uint64_t full_s[SLOTS], empty_s[SLOTS];
    __shared__ int abort_s;
    volatile int *abort_flag = &abort_s;
    const uint32_t full = smem_u32(full_s), empty = smem_u32(empty_s);
    auto load_group = [&](int it) { stream_load<MULTI>(p, rb, it, ring + (size_t)(it % SLOTS) * p.slot_bytes, full + 8 * (it % SLOTS)); };
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
        if (landed) {
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

// Q4_0.  The MMA's eight columns are the batch's NV vectors times 8 / NV blocks of 32 k: column j NV + v of the B operand is
// vector v where k lies in block j of a run of 8 / NV and zero elsewhere, so one accumulator collects the run's blocks side by
// side, exactly as accumulators of their own would, and scales are read and multiplied in once per run.  The order of k within a
// block is free, so a thread's share of a block is four neighbouring bytes: two blocks and their scales are nine aligned words.
// About 26 warp instructions per 16 x 32 weights at one vector (40 with an accumulator per block and 2-byte loads).  The quarters'
// sums are collected by one of the four warps, in turn, and the others go on.
// Rows of K / 32 * 18 bytes start in the same few banks where that is an even number of 16-byte pieces (K a multiple of 512): there a
// group comes as a box 16 bytes wider than the matrix, whose rows land an odd number of pieces apart.
// 262144 rows at m = 1, an accumulator per block / runs / runs and the box: K = 1536 57.4 / 46.1 / 44.7 us, K = 1024 57.2 / 37.0 / 32.8,
// K = 2048 147 (small-batch kernel) / 122 / 58.2; m = 2, K = 1536 59.2 / - / 45.3; 131072 rows, m = 4, K = 2048 75.6 / - / 33.9.
template <typename OutT, int UPQ, int NV, bool MULTI>
__global__ void __launch_bounds__(NT, 1) qgemv_q4_0_stream_kernel(const __grid_constant__ StreamParams p, const __grid_constant__ CUtensorMap w_map) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int BPR = 8 / NV, NRED = 4;   // blocks per run; buffers of sums
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int rg = warp & 3, kq = warp >> 2;
    lc_pdl_trigger();
    const uint32_t rb = (uint32_t)p.nb * 18u;
    const uint32_t base_a = (smem_u32(smem) + 127u) & ~127u;
    uint8_t *base = smem + (base_a - smem_u32(smem));
    float *red = reinterpret_cast<float *>(base);                    // [NRED][4 row groups][4 quarters][NV][16 rows]
    uint8_t *ring = base + NRED * 256 * NV * 4;                      // [slots][slot_bytes]
    const int my_groups = (p.groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    __shared__ __align__(8) uint64_t full_s[SLOTS], empty_s[SLOTS], summed_s[NRED * 4];
    __shared__ int abort_s;
    volatile int *abort_flag = &abort_s;
    const uint32_t full = smem_u32(full_s), empty = smem_u32(empty_s), summed = smem_u32(summed_s);
    auto load_group = [&](int it, int s) {
        if (MULTI || p.pitch == (int)rb) {
            stream_load<MULTI>(p, rb, it, ring + (size_t)s * p.slot_bytes, full + 8 * s);
            return;
        }
        mbar_arrive_expect_tx(full + 8 * s, (uint32_t)(GROUP_ROWS * p.pitch));
        tma_load_2d(smem_u32(ring) + (uint32_t)(s * p.slot_bytes), &w_map, 0, ((int)blockIdx.x + it * (int)gridDim.x) * GROUP_ROWS, full + 8 * s);
    };
    // the weights of the first groups do not depend on the previous kernel
    if (tid == NW * 32) {
        for (int s = 0; s < SLOTS; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, NW);
        }
        for (int s = 0; s < NRED * 4; s++) mbar_init(summed + 8 * s, 4);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int it = 0; it < p.slots && it < my_groups; it++) load_group(it, it);
    }
    lc_pdl_wait();
    bool alive = true;   // no wait of this warp has run out
    auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool {
        if (alive && !mbar_wait_warp(bar, parity, STREAM_WAIT_LIMIT)) {
            alive = false;
            *abort_flag = 1;
        }
        return alive;
    };
    if (warp == NW) {
        __syncthreads();
        uint32_t par = 0;
        for (int it = p.slots, s = 0; it < my_groups; it++) {
            if (!warp_wait(empty + 8 * s, par)) break;
            if (lane == 0) load_group(it, s);
            __syncwarp();
            if (++s == p.slots) { s = 0; par ^= 1u; }
        }
    } else {
        // this warp's quarter of K: blocks b0 .. b0 + nblk - 1 (a multiple of four), in runs
        constexpr int RUNS = UPQ * 4 < BPR ? 1 : (UPQ * 4 + BPR - 1) / BPR;
        const int nu = p.K / UNIT_K, upq = (nu + 3) / 4;
        const int b0 = min(kq * upq, nu) * 4, nblk = min(nu * 4 - b0, upq * 4);
        // Thread (g, t) is column g: it holds vector g % NV in block g / NV of a run.  Part 0 of a block is k 0 .. 15, part 1 the others.
        uint32_t breg[UPQ * 8][2];
#pragma unroll
        for (int r = 0; r < RUNS; r++) {
            uint2 x[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};
            if (BPR * r + g / NV < nblk && g % NV < p.m) {
#pragma unroll
                for (int part = 0; part < 2; part++)
                    x[part] = *reinterpret_cast<const uint2 *>(p.x + (size_t)(g % NV) * p.K + (b0 + BPR * r + g / NV) * 32 + 16 * part + 4 * t);
            }
#pragma unroll
            for (int j = 0; j < BPR; j++)
#pragma unroll
                for (int part = 0; part < 2; part++) {   // bytes 4t, 4t + 2 pair up in a register, and so do 4t + 1, 4t + 3
                    const int e = 2 * (BPR * r + j) + part;
                    if (e < UPQ * 8) {
                        breg[e][0] = g / NV == j ? __byte_perm(x[part].x, x[part].y, 0x5410) : 0u;
                        breg[e][1] = g / NV == j ? __byte_perm(x[part].x, x[part].y, 0x7632) : 0u;
                    }
                }
        }
        __syncthreads();   // the barriers are ready
        uint32_t par = 0;
        for (int it = 0, s = 0; it < my_groups; it++) {
            const bool landed = warp_wait(full + 8 * s, par);
            // (a group starts at a multiple of 64 rows of 72 bytes or a multiple: its slot starts with its first row)
            const uint32_t r0 = smem_u32(ring) + (uint32_t)(s * p.slot_bytes) + (uint32_t)((rg * 16 + g) * p.pitch) + (uint32_t)b0 * 18u;
            const uint32_t row_a[2] = {r0, r0 + 8u * (uint32_t)p.pitch};
            // Sums of rows g, g + 8 and the vectors of columns 2t, 2t + 1 (the same vector twice at NV = 1: one sum).
            float sum[2][2] = {};
            // this thread's columns' block within a run
            const uint32_t d_off = NV == 1 ? 36u * t : NV == 2 ? 18u * t : NV == 4 ? 18u * (t >> 1) : 0u;
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            if (landed) {
#pragma unroll
                for (int pr = 0; pr < UPQ * 2; pr++) {   // two blocks
                    if (2 * pr >= nblk) break;
                    uint32_t wq[2][2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const uint32_t a = row_a[i] + 4 * t + 36 * pr;
                        wq[0][i] = __byte_perm(lds32(a), lds32(a + 4), 0x5432);
                        wq[1][i] = lds32(a + 20);
                    }
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int blk = 2 * pr + e;
                        if (blk % BPR == 0) c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
                        for (int part = 0; part < 2; part++) {
                            const uint32_t a[4] = {codes_f16<4, 8>(wq[e][0], part), codes_f16<4, 8>(wq[e][1], part),
                                                   codes_f16<4, 8>(wq[e][0] >> 8, part), codes_f16<4, 8>(wq[e][1] >> 8, part)};
                            mma16816(c, a, breg[2 * blk + part][0], breg[2 * blk + part][1]);
                        }
                        // the run is complete (at NV = 1 a quarter may end inside one: its other blocks' sums are zero, their scales not
                        // this quarter's)
                        if (blk % BPR == BPR - 1 || (NV == 1 && blk % 4 == 3 && (blk == UPQ * 4 - 1 || blk == nblk - 1))) {
                            const int first = blk / BPR * BPR;
                            if (NV > 1 || first + 2 * t < nblk) {
#pragma unroll
                                for (int i = 0; i < 2; i++) {
                                    const float d = lds_f16(row_a[i] + 18 * first + d_off);
                                    sum[i][0] = fmaf(d, c[2 * i], sum[i][0]);
                                    if (NV == 1) sum[i][0] = fmaf(lds_f16(row_a[i] + 18 * first + 18 + d_off), c[2 * i + 1], sum[i][0]);
                                    else sum[i][1] = fmaf(d, c[2 * i + 1], sum[i][1]);
                                }
                            }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * s);
            // Threads of a quad that hold other blocks of the same vectors.
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int v = 0; v < (NV == 1 ? 1 : 2); v++) {
                    if (NV <= 2) sum[i][v] += __shfl_xor_sync(0xffffffffu, sum[i][v], 1);
                    if (NV <= 4) sum[i][v] += __shfl_xor_sync(0xffffffffu, sum[i][v], 2);
                }
            // Four buffers: between two writes of one, each warp has been the one that collects, so it has seen every warp past the
            // reads of the first.
            float *rd = red + ((it & (NRED - 1)) * 4 + rg) * 64 * NV;
            const uint32_t bar = summed + 8 * ((it & (NRED - 1)) * 4 + rg);
            float *mine = rd + kq * 16 * NV + g;
            if (NV == 1) {
                if (t < 2) mine[8 * t] = t ? sum[1][0] : sum[0][0];
            } else if (NV == 2) {
                mine[16 * (t & 1) + 8 * (t >> 1)] = (t & 1) ? ((t >> 1) ? sum[1][1] : sum[0][1]) : ((t >> 1) ? sum[1][0] : sum[0][0]);
            } else if (NV == 4) {
                mine[32 * (t & 1) + 8 * (t >> 1)] = (t >> 1) ? sum[1][0] : sum[0][0];
                mine[32 * (t & 1) + 16 + 8 * (t >> 1)] = (t >> 1) ? sum[1][1] : sum[0][1];
            } else {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    mine[32 * t + 8 * i] = sum[i][0];
                    mine[32 * t + 16 + 8 * i] = sum[i][1];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
            if ((it & 3) == kq && warp_wait(bar, (uint32_t)((it / NRED) & 1)) && landed) {
                const int gl = (int)blockIdx.x + it * (int)gridDim.x, mi = MULTI ? gl / p.gpm : 0, grp = gl - mi * p.gpm;
                const int row = grp * GROUP_ROWS + rg * 16 + (lane & 15);
#pragma unroll
                for (int o = lane; o < 16 * NV; o += 32) {
                    const float v = ((rd[o] + rd[16 * NV + o]) + rd[32 * NV + o]) + rd[48 * NV + o];
                    if (row < p.n && (o >> 4) < p.m) store_c(reinterpret_cast<OutT *>(p.out[mi]) + (size_t)(o >> 4) * p.n + row, v * 512.0f);
                }
            }
            if (++s == p.slots) { s = 0; par ^= 1u; }
        }
    }
    __syncthreads();
    if (*abort_flag) tc_wait_expired(p.status, LC_DEV_STATUS_WAIT_EXPIRED, tid);
}

template <typename OutT, int UPQ, int NV, bool MULTI>
int launch_q4_0(lc_kernels *k, lc_batch *b, const StreamParams &p, const CUtensorMap &w_map, size_t smem) {
    auto kern = qgemv_q4_0_stream_kernel<OutT, UPQ, NV, MULTI>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    const int grid = p.groups < k->ctx->sm_count ? p.groups : k->ctx->sm_count;
    LC_LAUNCH_CHECKED(lc_launch(kern, dim3(grid), dim3(NT), smem, b, p, w_map));
    b->dispatch_count++;
    return LC_OK;
}
template <typename OutT, int UPQ>
int launch_q4_0_v(lc_kernels *k, lc_batch *b, const StreamParams &p, const CUtensorMap &w_map, size_t smem) {
    if (p.groups > p.gpm) return launch_q4_0<__half, UPQ, 1, true>(k, b, p, w_map, smem);   // (groups are f16 and one vector)
    switch (p.m) {
        case 1: return launch_q4_0<OutT, UPQ, 1, false>(k, b, p, w_map, smem);
        case 2: return launch_q4_0<OutT, UPQ, 2, false>(k, b, p, w_map, smem);
        case 3:
        case 4: return launch_q4_0<OutT, UPQ, 4, false>(k, b, p, w_map, smem);
        default: return launch_q4_0<OutT, UPQ, 8, false>(k, b, p, w_map, smem);
    }
}
template <typename OutT>
int launch_q4_0_u(lc_kernels *k, lc_batch *b, const StreamParams &p, const CUtensorMap &w_map, size_t smem) {
    switch ((p.K / UNIT_K + 3) / 4) {
        case 1: return launch_q4_0_v<OutT, 1>(k, b, p, w_map, smem);
        case 2: return launch_q4_0_v<OutT, 2>(k, b, p, w_map, smem);
        case 3: return launch_q4_0_v<OutT, 3>(k, b, p, w_map, smem);
        default: return launch_q4_0_v<OutT, 4>(k, b, p, w_map, smem);
    }
}
// K <= 2048
int stream_q4_0(bool f32out, lc_kernels *k, lc_batch *b, StreamParams &p) {
    const uint32_t rb = (uint32_t)p.nb * 18u;
    const bool multi = p.groups > p.gpm;
    CUtensorMap w_map = {};
    p.pitch = (int)rb;
    if (!multi && rb % 32 == 0 && lc_wider_rows_map(&w_map, k->test_map_refused, p.w[0], rb, (uint32_t)p.n, GROUP_ROWS)) p.pitch = (int)rb + 16;
    p.slot_bytes = (GROUP_ROWS * p.pitch + 16 + 127) / 128 * 128;
    const int nv = p.m <= 2 ? p.m : p.m <= 4 ? 4 : 8;
    auto bytes = [&](int slots) { return (size_t)128 + 4 * 256 * nv * sizeof(float) + (size_t)slots * p.slot_bytes; };
    p.slots = bytes(SLOTS) + 512 <= k->ctx->smem_optin ? SLOTS : SLOTS - 1;   // (the barriers are static)
    const size_t smem = bytes(p.slots);
    if (smem + 512 > k->ctx->smem_optin) return -1;
    return f32out ? launch_q4_0_u<float>(k, b, p, w_map, smem) : launch_q4_0_u<__half>(k, b, p, w_map, smem);
}

template <typename OutT, int UPQ, bool MULTI>
int launch_tq2_0_um(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    auto kern = qgemv_tq2_0_stream_kernel<OutT, UPQ, MULTI>;
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(kern, optin, b->ctx, smem));
    const int grid = p.groups < k->ctx->sm_count ? p.groups : k->ctx->sm_count;
    LC_LAUNCH_CHECKED(lc_launch(kern, dim3(grid), dim3(NT), smem, b, p));
    b->dispatch_count++;
    return LC_OK;
}
template <typename OutT, int UPQ>
int launch_tq2_0_u(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    return p.groups > p.gpm ? launch_tq2_0_um<OutT, UPQ, true>(k, b, p, smem) : launch_tq2_0_um<OutT, UPQ, false>(k, b, p, smem);
}

template <typename OutT>
int launch_tq2_0(lc_kernels *k, lc_batch *b, const StreamParams &p, size_t smem) {
    const int upq = (p.K / UNIT_K + 3) / 4;
    switch (upq) {
        case 1: return launch_tq2_0_u<OutT, 1>(k, b, p, smem);
        case 2: return launch_tq2_0_u<OutT, 2>(k, b, p, smem);
        case 3: return launch_tq2_0_u<OutT, 3>(k, b, p, smem);
        default: return launch_tq2_0_u<OutT, 0>(k, b, p, smem);
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
    // worth it only when every SM gets a few groups to stream
    const int gpm = (int)((n + GROUP_ROWS - 1) / GROUP_ROWS);
    if ((int64_t)gpm * count < 2 * k->ctx->sm_count) return -1;
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
    p.gpm = gpm;
    p.status = k->dev_status;
    p.groups = p.gpm * count;
    if (fmt == FMT_Q4_0) return kk <= 16 * UNIT_K ? stream_q4_0(f32out, k, b, p) : -1;
    p.xs = (int)kk * 2 + 16;
    p.slot_bytes = (int)(((size_t)GROUP_ROWS * p.nb * bb + 15 + 15) / 16 * 16 + 16);
    const size_t smem = (size_t)8 * p.xs + 2 * NW * 32 * 16 + (size_t)SLOTS * p.slot_bytes;
    if (smem + 256 > k->ctx->smem_optin) return -1;   // (the barriers are static)
    return f32out ? launch_tq2_0<float>(k, b, p, smem) : launch_tq2_0<__half>(k, b, p, smem);
}

int lc_qgemv_mma_stream(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                        lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    const lc_buf *ws[1] = {weight};
    lc_buf *os[1] = {output};
    return lc_qgemv_mma_stream_group(fmt, f32out, k, b, input, 1, ws, os, m, kk, n);
}
