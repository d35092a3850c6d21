// Tensor-core decode attention over TurboQuant codes: tq2 / tq3 / tq4, head_dim 128 / 256 / 512, 8 q-heads of a kv-head
// per CTA.  Same contract, grid and split-K partial layout as tq_attn_split_kernel (attention_tq.cu), which serves what is
// left: head_dim 64, operands at odd offsets, very short rings.
//
// With 8 q-heads sharing every K/V row the CUDA-core kernel needs 16 x head_dim FMAs per key, which binds long before HBM
// does.  Here both contractions run on tensor cores, with operands built in registers from the packed codes:
//   * a shared-memory table maps one field of code bits (8 bits: four tq2 or two tq4 codes; 6 or 4 bits: two tq3 or tq2 codes) to
//     f16 levels with a single 8-byte load; it is replicated 16 times so that the lookups of a half-warp never collide;
//   * S^T[16 keys x 8 heads] = K[16 x HD] . RQ^T: the contraction index (dims) is free to permute, so thread (g, t) of a
//     warp feeds the MMA with the HD / 4 dims held in its own quarter of the code bytes of keys g, g + 8;
//   * O^T[HD dims x 8 heads] += V^T[HD x 16 keys] . P: the A operand wants (dim; two adjacent keys) per register, so
//     thread (g, t) takes its eighth of the code bytes of keys 2t, 2t + 1, 2t + 8, 2t + 9 and puts the codes of adjacent keys side by
//     side before the lookup, whose two registers are then operand registers (attn_tile); at head_dim 512 the table entries of adjacent keys
//     are paired by byte permutes.  P reaches the B operand through one movmatrix transpose per 8 keys.
// A warp step is KT = 32 keys (16 at head_dim 512): two independent sets of accumulation chains, and the softmax, the
// running-maximum shuffles and the refill arithmetic are paid once per 32 keys.  Codes stream through a per-warp
// cp.async ring; consecutive lanes copy consecutive 16-byte pieces, so a tile of one kv-head is one contiguous read.
//
// What bounds it: instruction issue and fetch, not a pipe (ncu, tq2, 64 lanes x 8192 keys: 33 warp instructions per key, 0.46 issued per cycle and
// scheduler; ALU 35 %, tensor 26 %, shared memory 47 % busy; 12 or 16 warps with the query in shared memory are no
// faster).  At head_dim 256 a key takes an SM 15.5 cycles at tq2, 30 at tq4.  64 lanes x 8192 keys: 57 -> 47 -> 40 us (tq2), 480 (the CUDA-core kernel)
// -> 85 -> 80 us (tq4); 64 ragged lanes up to 8192 keys at tq4: 259 -> 47 -> 44 us.
//
// Precision.  The query is split into an f16 and the f16 of the remainder (two MMAs), because logits reach |q||k| ~ head_dim
// at softmax scale 1.  The table holds each level as an f16 and the f16 of its remainder, and so is P (three MMAs per contraction
// step): the result is within 6e-6 of its norm against 64 bits.  Only tq2 at head_dim 256 makes do with one f16 each, P as it is and
// levels / gamma, gamma searched (1024 mantissas) so that all four are f16-representable to ~2e-6 and folded into the row
// norms in f32: 2e-4, mostly P's.  (64 lanes x 8192 keys of 128 took 31.6 us in that form, 46.8 in this one and 164 on CUDA cores,
// whose error was 1e-6; behind an f16 output the single f16 showed as 3.0e-4 for 2.1e-4.)
#include <math.h>

#include "attention_tq_tile.cuh"

namespace {

// QUEUE: the queue form (TqAttnParams::queue_chunk), an instantiation of its own so that the others' code stays short.
template <typename C, bool QUEUE>
__global__ void __launch_bounds__(C::NT) tq_attn_mma_kernel(const TqAttnParams p) {
    constexpr int HD = C::HD, CB = C::CB, NW = C::NW, NT = C::NT, KT = C::KT, NS = C::NS, DPL = C::DPL;
    lc_pdl_trigger();
    if (p.cluster_merge) cluster_arrive_relaxed();   // awaited before the first store to a peer's shared memory
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t base_a = smem_u32(smem);
    uint2 *lut = reinterpret_cast<uint2 *>(smem);                       // [NENT][16 copies]
    float *rq_s = reinterpret_cast<float *>(smem + C::LUT_BYTES);       // [NS][32 lanes][4] rotated, scaled query
    __shared__ uint32_t q_first[QUEUE ? LC_ATTN_QUEUE_LANES + 1 : 1];               // queue form: first item of each lane
    __shared__ uint32_t q_pos[QUEUE ? LC_ATTN_QUEUE_LANES : 1];                     // and its position
    __shared__ uint32_t q_ticket;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t gchunks = (p.group + G - 1) / G;
    const uint32_t kv_head = blockIdx.y / gchunks, gchunk = blockIdx.y - kv_head * gchunks;
    const int gvalid = min((int)G, (int)(p.group - gchunk * G));
    const uint32_t qh0 = kv_head * p.group + gchunk * G;

    // ---- before the dependency wait: everything that depends on the codec's levels only (a constant operand): gamma and
    //      the table.  A CTA that becomes resident while its predecessor drains does this part for free (and where there is no
    //      predecessor, built while the first loads were on their way it took as long). ----
    const float gamma = attn_table<C>(p.levels, lut, lane, warp);
    const uint32_t lut_lane = base_a + (uint32_t)(lane & (LUT_COPIES - 1)) * 8u;

    // Codes and norms of keys below the lanes' positions were written by earlier steps; only the key at the position
    // itself comes from the predecessor.  A caller that also guarantees that `positions` was written before the
    // predecessor kernels started (the decode step: it is an input of the step) sets early_kv, and the first tiles'
    // copies are then in flight while the predecessor finishes.
    const bool early = p.early_kv != 0u && p.positions != nullptr && p.row_positions == 0u && !QUEUE;
    if (!early && !(QUEUE && p.early_kv)) lc_pdl_wait();

    // keys [win_start, seq_len) of a lane
    auto lane_range = [&](uint32_t li, uint32_t &pos, uint32_t &seq_len, uint32_t &win_start, bool report, bool in_smem) {
        if (p.positions) {
            pos = in_smem ? q_pos[li] : p.positions[li];
            seq_len = pos + 1u;
            if (p.ring == 0u && seq_len > p.lane_capacity) {   // never read past the lane's rows
                seq_len = p.lane_capacity;
                if (report && p.status && threadIdx.x == 0) atomicExch(p.status, LC_DEV_STATUS_POSITION);
            }
        } else {
            pos = p.current_pos + (p.row_positions ? li : 0u);
            seq_len = min(p.kv_len, pos + 1u);
        }
        win_start = (p.window > 0u && pos + 1u > p.window) ? (pos + 1u - p.window) : 0u;
    };
    uint32_t n_items = 0;
    if (QUEUE) {
        for (uint32_t li = threadIdx.x; li < p.n_lanes; li += NT) {
            uint32_t pos, seq_len, ws;
            lane_range(li, pos, seq_len, ws, false, false);
            q_pos[li] = pos;
            const uint32_t n = seq_len > ws ? seq_len - ws : 0u;
            q_first[li + 1] = lc_attn_items(n, p.queue_chunk);   // (an empty lane is one item and stores zeros)
        }
        if (threadIdx.x == 0) q_first[0] = 0;
        __syncthreads();
        if (warp == 0) {   // prefix sums
            uint32_t carry = 0;
            for (uint32_t l0 = 0; l0 < p.n_lanes; l0 += 32) {
                const uint32_t li = l0 + lane;
                uint32_t v = li < p.n_lanes ? q_first[li + 1] : 0u;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                v += carry;
                if (li < p.n_lanes) q_first[li + 1] = v;
                carry = __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        n_items = q_first[p.n_lanes];
        if (p.early_kv) lc_pdl_wait();
    }
    // A CTA's first item is its own number; it draws the others one after the other.
    uint32_t item = blockIdx.x;
    uint32_t ticket = 0;   // thread 0
    auto draw = [&]() { ticket = atomicAdd(&p.counters[blockIdx.y], 1u); };

    // The item at hand: keys [k_begin, k_end) of lane lane_idx, its part number `split`.
    uint32_t lane_idx = blockIdx.z, split = blockIdx.x, pos = 0, k_begin = 0, k_end = 0;
    auto next_item = [&]() -> bool {
        if (QUEUE) {
            if (item >= n_items) return false;
            uint32_t before = 0;   // lanes whose items all come first
            for (uint32_t l0 = 0; l0 < p.n_lanes; l0 += 32)
                before += __popc(__ballot_sync(0xffffffffu, l0 + lane < p.n_lanes && q_first[l0 + lane + 1] <= item));
            lane_idx = before;
            split = item - q_first[lane_idx];
        }
        uint32_t seq_len, win_start;
        lane_range(lane_idx, pos, seq_len, win_start, true, QUEUE);
        const uint32_t n_keys = seq_len > win_start ? seq_len - win_start : 0u;
        uint32_t per;
        if (QUEUE) {
            per = lc_attn_item_keys(n_keys, p.queue_chunk);
        } else {
            per = (n_keys + p.n_splits - 1) / p.n_splits;
            per = (per + (KT - 1)) & ~(uint32_t)(KT - 1);
        }
        k_begin = win_start + split * per;
        k_end = min(seq_len, k_begin + per);
        return true;
    };

    // Each warp keeps DEPTH - 1 tiles of codes in flight in its own ring: KT rows of K, then KT rows of V.
    const uint32_t ring_a = base_a + (uint32_t)C::RING_OFF + (uint32_t)(warp * C::DEPTH) * C::STAGE;
    auto slot_of = [&](uint32_t t0, uint32_t off) -> size_t {
        uint32_t r = p.ring ? t0 % p.ring : t0;   // (ring >= KT)
        if (t0 + off < k_end) r += off;           // t0 is always a valid key
        if (p.ring && r >= p.ring) r -= p.ring;
        return ((size_t)lane_idx * p.lane_capacity + r) * p.n_kv + kv_head;
    };
    auto issue = [&](uint32_t t0, int stage) {
        constexpr int CPR = CB / 16, PER_LANE = KT * CPR / 32;
        const uint32_t dst = ring_a + (uint32_t)stage * C::STAGE;
        const uint32_t r0 = p.ring ? t0 % p.ring : t0;
        if (t0 + KT <= k_end && (p.ring == 0u || r0 + KT <= p.ring)) {   // the usual tile: KT rows at one stride
            const size_t s0 = ((size_t)lane_idx * p.lane_capacity + r0) * p.n_kv + kv_head;
            const uint8_t *kb = p.kc + s0 * CB, *vb = p.vc + s0 * CB;
            const uint32_t rs = p.n_kv * (uint32_t)CB;
#pragma unroll
            for (int i = 0; i < PER_LANE; i++) {
                const uint32_t c = (uint32_t)(i * 32 + lane), row = c / CPR, off = (c - row * CPR) * 16u;
                cp_async16(dst + row * C::KRS + off, kb + row * rs + off);
                cp_async16(dst + KT * C::KRS + row * C::VRS + off, vb + row * rs + off);
            }
        } else {
#pragma unroll 1
            for (int i = 0; i < PER_LANE; i++) {
                const uint32_t c = (uint32_t)(i * 32 + lane), row = c / CPR, off = (c - row * CPR) * 16u;
                const size_t s = slot_of(t0, row);
                cp_async16(dst + row * C::KRS + off, p.kc + s * CB + off);
                cp_async16(dst + KT * C::KRS + row * C::VRS + off, p.vc + s * CB + off);
            }
        }
    };
    // this lane's norms of a tile: key norm of key `lane`, value norm of key `lane` (KT = 16: lanes 16-31 repeat)
    auto load_norms = [&](uint32_t t0, __half &nk, __half &nv) {
        if (t0 < k_end) {
            const size_t s = slot_of(t0, (uint32_t)lane & (KT - 1));
            nk = p.kn[s];
            nv = p.vn[s];
        }
    };
    uint32_t t_issue = 0;
    __half nk_raw = __float2half(0.f), nv_raw = nk_raw;
    auto start_item = [&](int issued) {   // the item's first tiles but the `issued` ones
#pragma unroll
        for (int i = 0; i < C::DEPTH - 1; i++) {
            if (i >= issued) {
                if (t_issue < k_end) issue(t_issue, i);
                cp_async_commit();
                t_issue += NW * KT;
            }
        }
        load_norms(k_begin + warp * KT, nk_raw, nv_raw);
    };
    // warp w's share of the query: head w's dims DPL lane .., as they are
    const bool have_frag = p.qfrag != nullptr;   // the launch that wrote q left the fragments ready (group % 8 == 0)
    uint4 q_raw[DPL / 4];
    auto load_query = [&]() {
        if (have_frag || warp >= gvalid) return;
        const size_t q_row = ((size_t)lane_idx * p.n_q + qh0 + warp) * HD + DPL * lane;
#pragma unroll
        for (int i = 0; i < DPL; i += 4) {
            if (p.fused_q) {
                const uint2 v = *reinterpret_cast<const uint2 *>(p.q + q_row + i);
                q_raw[i / 4].x = v.x;
                q_raw[i / 4].y = v.y;
            } else {
                q_raw[i / 4] = *reinterpret_cast<const uint4 *>(p.rq + q_row + i);
            }
        }
    };
    bool more = next_item();
    t_issue = k_begin + warp * KT;
    // With early_kv the first tiles leave before the dependency wait, up to the tile that holds the key the
    // predecessor is writing (position pos: the last key of the last split); that tile and the ones after it follow
    // the wait.  Groups are committed in tile order either way.
    int issued = 0;
    if (early) {
#pragma unroll
        for (int i = 0; i < C::DEPTH - 1; i++) {
            if (issued == i && !(t_issue <= pos && pos < t_issue + KT)) {
                if (t_issue < k_end) issue(t_issue, i);
                cp_async_commit();
                t_issue += NW * KT;
                issued = i + 1;
            }
        }
        lc_pdl_wait();
    }
    if (more) {
        start_item(issued);
        load_query();
    }

    while (more) {
        // ---- after the wait: the query.  B fragments: thread (g, t) holds head g, dims t HD/4 + 4s + {0,1} and + {2,3}.
        //      It is the one operand f16 cannot hold well enough: a high f16 part and the f16 of the remainder. ----
        constexpr int NQ = C::QSMEM ? 1 : NS;
        uint32_t bq[NQ][2], bql[NQ][2];
        if (C::QSMEM && have_frag) {
            const uint4 *src = p.qfrag + ((size_t)lane_idx * (p.n_q >> 3) + (qh0 >> 3)) * (NS * 32);
            for (int e = threadIdx.x; e < NS * 32; e += NT) *reinterpret_cast<uint4 *>(rq_s + e * 4) = src[e];
        } else if (!C::QSMEM && have_frag) {
            const uint4 *src = p.qfrag + ((size_t)lane_idx * (p.n_q >> 3) + (qh0 >> 3)) * (NS * 32) + lane;
#pragma unroll
            for (int s = 0; s < NQ; s++) {
                const uint4 v = src[s * 32];
                bq[s][0] = v.x;
                bq[s][1] = v.y;
                bql[s][0] = v.z;
                bql[s][1] = v.w;
            }
        } else if (warp < G) {   // warp w rotates and scales head w
            float x[DPL];
#pragma unroll
            for (int i = 0; i < DPL; i++) x[i] = 0.f;
            if (warp < gvalid) {
                if (p.fused_q) {
#pragma unroll
                    for (int i = 0; i < DPL; i += 4) {
                        const uint4 raw = q_raw[i / 4];
                        const float4 sg = *reinterpret_cast<const float4 *>(p.signs + DPL * lane + i);
                        const float2 f0 = unpack_h2(raw.x), f1 = unpack_h2(raw.y);
                        x[i] = f0.x * sg.x;
                        x[i + 1] = f0.y * sg.y;
                        x[i + 2] = f1.x * sg.z;
                        x[i + 3] = f1.y * sg.w;
                    }
                    warp_fwht<DPL>(x, lane);
                    const float f = p.scale / sqrtf((float)HD);
#pragma unroll
                    for (int i = 0; i < DPL; i++) x[i] *= f;
                } else {
#pragma unroll
                    for (int i = 0; i < DPL; i += 4) {
                        const uint4 r = q_raw[i / 4];
                        x[i] = __uint_as_float(r.x) * p.scale;
                        x[i + 1] = __uint_as_float(r.y) * p.scale;
                        x[i + 2] = __uint_as_float(r.z) * p.scale;
                        x[i + 3] = __uint_as_float(r.w) * p.scale;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < DPL; i += 4) {   // dim d = t HD/4 + 4s + e is element e of entry [s][lane 4 head + t]
                const int d = DPL * lane + i;
                *reinterpret_cast<float4 *>(rq_s + (((d % (HD / 4)) / 4) * 32 + warp * 4 + d / (HD / 4)) * 4) =
                    make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            }
        }
        __syncthreads();   // the rotated query is in place; so is every copy of the table
        if (C::QSMEM) {
            if (!have_frag)
            for (int e = threadIdx.x; e < NS * 32; e += NT) {   // in place: entry e is read and written by one thread
                const float4 r = *reinterpret_cast<const float4 *>(rq_s + e * 4);
                uint4 v;
                split_h2(r.x, r.y, v.x, v.z);
                split_h2(r.z, r.w, v.y, v.w);
                *reinterpret_cast<uint4 *>(rq_s + e * 4) = v;
            }
            __syncthreads();
        } else if (!have_frag) {
#pragma unroll
            for (int s = 0; s < NQ; s++) {
                const float4 r = *reinterpret_cast<const float4 *>(rq_s + (s * 32 + lane) * 4);
                split_h2(r.x, r.y, bq[s][0], bql[s][0]);
                split_h2(r.z, r.w, bq[s][1], bql[s][1]);
            }
        }
        const uint32_t q_a = base_a + (uint32_t)C::LUT_BYTES + (uint32_t)lane * 16u;

        // ---- main loop: each warp takes every 8th tile of this split ----
        AttnAcc<C> acc;
        acc.clear();
        float(&m_run)[2] = acc.m_run, (&l_part)[2] = acc.l_part;

        int stage = 0;
        for (uint32_t t0 = k_begin + warp * KT; t0 < k_end; t0 += NW * KT) {
            if (QUEUE && threadIdx.x == 0 && t0 + NW * KT >= k_end) draw();   // as late as a tile hides the round trip
            cp_async_wait<C::DEPTH - 2>();   // tile t0 is the oldest group in flight
            __syncwarp();                    // ... for every lane; and every lane is done with the tile before
            const float nk = __half2float(nk_raw) * gamma, nv = __half2float(nv_raw) * gamma;
            load_norms(t0 + NW * KT, nk_raw, nv_raw);
            {
                const int st_fill = stage == 0 ? C::DEPTH - 1 : stage - 1;
                if (t_issue < k_end) issue(t_issue, st_fill);
                cp_async_commit();
                t_issue += NW * KT;
            }
            const uint32_t ka = ring_a + (uint32_t)stage * C::STAGE, va = ka + KT * C::KRS;
            stage = stage + 1 == C::DEPTH ? 0 : stage + 1;

            attn_tile<C>(acc, ka, va, t0, k_end, nk, nv, bq, bql, q_a, lut_lane, lane);
        }

        if (QUEUE && threadIdx.x == 0) {
            if (k_begin >= k_end) draw();
            if (ticket == n_items - 1u) p.counters[blockIdx.y] = 0u;   // every CTA has drawn its last: zero again for the next launch
            q_ticket = gridDim.x + ticket;
        }

        // ---- merge the warps that had keys; query and ring memory is reused for their accumulators.  A step of the decode
        //      model comes here after one or two tiles per warp, with this code cold in the instruction cache: it is
        //      kept short (with the finish below 12.4 -> 10.1 us for 64 lanes x 512 keys, 9.5 -> 7.9 us for one lane). ----
#pragma unroll
        for (int h = 0; h < 2; h++) {
            l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 4);
            l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 8);
            l_part[h] += __shfl_xor_sync(0xffffffffu, l_part[h], 16);
        }
        float *acc_s = reinterpret_cast<float *>(smem + C::LUT_BYTES);   // [NW][NS][32 lanes][4]: fragment order
        float *m_s = reinterpret_cast<float *>(smem + C::TAIL_OFF);      // [NW][G]
        float *l_s = m_s + NW * G;
        float *ml_s = l_s + NW * G;                                      // [ROWS][2]
        float *cpart = ml_s + 2 * C::ROWS;                               // merged, unnormalised rows (cp_index)
        if (g == 0) *reinterpret_cast<float2 *>(m_s + warp * G + 2 * t) = make_float2(m_run[0], m_run[1]);
        __syncthreads();   // every warp is done with its ring, and its maximum is known
        const uint32_t tiles_all = k_end > k_begin ? (k_end - k_begin + KT - 1) / KT : 0u;
        const int nwa = tiles_all < (uint32_t)NW ? (int)tiles_all : NW;
        {
            float g0 = -INFINITY, g1 = -INFINITY;
#pragma unroll
            for (int w = 0; w < NW; w++) {
                const float2 v = *reinterpret_cast<const float2 *>(m_s + w * G + 2 * t);
                g0 = fmaxf(g0, v.x);
                g1 = fmaxf(g1, v.y);
            }
            const float f0 = m_run[0] == -INFINITY ? 0.f : soft_exp<C::HILO>(m_run[0] - g0);
            const float f1 = m_run[1] == -INFINITY ? 0.f : soft_exp<C::HILO>(m_run[1] - g1);
            if (g == 0) *reinterpret_cast<float2 *>(l_s + warp * G + 2 * t) = make_float2(f0 * l_part[0], f1 * l_part[1]);
            if (warp < nwa) {
                float4 *dst = reinterpret_cast<float4 *>(acc_s) + warp * NS * 32 + lane;
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    const float4 v = acc.result(s);
                    dst[s * 32] = make_float4(v.x * f0, v.y * f1, v.z * f0, v.w * f1);
                }
            }
        }
        // Head h's row: of this CTA alone row h; in a cluster row (h / n) * n + split of CTA h mod n, which finishes head h.
        auto row_of = [&](int h) -> int { return p.cluster_merge ? (h / (int)p.n_splits) * (int)p.n_splits + (int)split : h; };
        auto peer_addr = [&](const float *a, int h) -> uint32_t { return cluster_addr(smem_u32(a), (uint32_t)h % p.n_splits); };
        if (p.cluster_merge) cluster_wait();   // (of the arrival at the start) every CTA of the cluster runs
        __syncthreads();
        if (threadIdx.x < G) {   // merged (max, sum) of head h
            const int h = threadIdx.x;
            float gmax = -INFINITY, gsum = 0.f;
#pragma unroll
            for (int w = 0; w < NW; w++) {
                gmax = fmaxf(gmax, m_s[w * G + h]);
                gsum += l_s[w * G + h];
            }
            float *dst = ml_s + 2 * row_of(h);
            if (p.cluster_merge)
                st_cluster_f2(peer_addr(dst, h), gmax, gsum);
            else
                *reinterpret_cast<float2 *>(dst) = make_float2(gmax, gsum);
        }
        const size_t part_row = HD + 2;
        const uint32_t it_lane = lane_idx, it_split = split;
        if (QUEUE) {   // what comes next, and its query on the way
            item = q_ticket;
            if (next_item()) load_query();
        }
        // where head h's partial of this split goes
        auto part_of = [&](int h, uint32_t sp) -> float * {
            const size_t qh = (size_t)it_lane * p.n_q + qh0 + h;
            return p.partial + (qh * p.n_splits + sp) * part_row;
        };
        // Thread (warp, lane) adds fragment position `lane` of its tiles s: heads 2t and 2t + 1 at dims (HD / 8) g + 2 s + 0, 1.
        {
            constexpr int TW = NS / NW;
            float4 sum[TW];
#pragma unroll
            for (int i = 0; i < TW; i++) sum[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 *src = reinterpret_cast<const float4 *>(acc_s) + warp * 32 + lane;
#pragma unroll
            for (int w = 0; w < NW; w++) {
#pragma unroll
                for (int i = 0; i < TW; i++) {
                    const float4 v = w < nwa ? src[(w * NS + i * NW) * 32] : make_float4(0.f, 0.f, 0.f, 0.f);
                    sum[i].x += v.x; sum[i].y += v.y; sum[i].z += v.z; sum[i].w += v.w;
                }
            }
            float *r0 = cpart + C::cp_index(row_of(2 * t), (HD / 8) * g), *r1 = cpart + C::cp_index(row_of(2 * t + 1), (HD / 8) * g);
            if (p.cluster_merge) {
                const uint32_t a0 = peer_addr(r0, 2 * t), a1 = peer_addr(r1, 2 * t + 1);
#pragma unroll
                for (int i = 0; i < TW; i++) {
                    st_cluster_f2(a0 + (uint32_t)(warp + i * NW) * 8u, sum[i].x, sum[i].z);
                    st_cluster_f2(a1 + (uint32_t)(warp + i * NW) * 8u, sum[i].y, sum[i].w);
                }
            } else {
#pragma unroll
                for (int i = 0; i < TW; i++) {
                    *reinterpret_cast<float2 *>(r0 + 2 * (warp + i * NW)) = make_float2(sum[i].x, sum[i].z);
                    *reinterpret_cast<float2 *>(r1 + 2 * (warp + i * NW)) = make_float2(sum[i].y, sum[i].w);
                }
            }
        }
        if (p.cluster_merge) {
            // The splits of this (lane, kv head) are one cluster, and every row this CTA finishes is in its own shared memory
            // after the barrier: nobody reads a peer's, so there is no second barrier.  One warp per head: the same arithmetic,
            // in the same order, as tq_attn_merge_kernel (attention_tq.cu).
            const int n = (int)p.n_splits;
            float4 sg[DPL / 4];   // (the load's round trip passes at the barrier)
            if (p.fused_q) {
#pragma unroll
                for (int i = 0; i < DPL / 4; i++) sg[i] = *reinterpret_cast<const float4 *>(p.signs + DPL * lane + 4 * i);
            }
            cluster_arrive_release();
            cluster_wait();
            for (int h = (int)split + n * warp; h < gvalid; h += n * NW) {
                const int row0 = (h / n) * n;
                const float2 ml = lane < n ? *reinterpret_cast<const float2 *>(ml_s + 2 * (row0 + lane)) : make_float2(-INFINITY, 0.f);
                float gmax = ml.x;
                gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 1));
                gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 2));
                gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 4));
                const float fl = ml.x == -INFINITY ? 0.f : expf(ml.x - gmax);   // (lanes past the eighth hold nothing)
                float gsum = 0.f, ov[DPL];
#pragma unroll
                for (int i = 0; i < DPL; i++) ov[i] = 0.f;
#pragma unroll 2
                for (int sp = 0; sp < n; sp++) {
                    const float f = __shfl_sync(0xffffffffu, fl, sp);
                    gsum += f * __shfl_sync(0xffffffffu, ml.y, sp);
#pragma unroll
                    for (int i = 0; i < DPL; i += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(cpart + C::cp_index(row0 + sp, DPL * lane + i));
                        ov[i] += f * v.x; ov[i + 1] += f * v.y; ov[i + 2] += f * v.z; ov[i + 3] += f * v.w;
                    }
                }
#pragma unroll
                for (int i = 0; i < DPL; i++) ov[i] = gsum > 0.f ? ov[i] / gsum : 0.f;
                const size_t qh = (size_t)it_lane * p.n_q + qh0 + h;
                if (!p.fused_q) {
#pragma unroll
                    for (int i = 0; i < DPL; i += 4)
                        *reinterpret_cast<float4 *>(p.out + qh * HD + DPL * lane + i) = make_float4(ov[i], ov[i + 1], ov[i + 2], ov[i + 3]);
                    continue;
                }
                // inverse rotation, 1/sqrt(d), signs
                warp_fwht<DPL>(ov, lane);
                const float inv = 1.0f / sqrtf((float)HD);
#pragma unroll
                for (int i = 0; i < DPL; i += 4) {
                    uint2 packed;
                    packed.x = pack_h2(ov[i] * inv * sg[i / 4].x, ov[i + 1] * inv * sg[i / 4].y);
                    packed.y = pack_h2(ov[i + 2] * inv * sg[i / 4].z, ov[i + 3] * inv * sg[i / 4].w);
                    *reinterpret_cast<uint2 *>(p.out_f16 + qh * HD + DPL * lane + i) = packed;
                }
            }
            return;
        }
        __syncthreads();   // the tile is complete; the ring is free
        more = QUEUE && item < n_items;
        if (more) {
            t_issue = k_begin + warp * KT;
            start_item(0);
        }
        // a merge launch follows (unless there is nothing to merge)
        for (int e = threadIdx.x; e < gvalid * (HD / 2); e += NT) {
            const int h = e / (HD / 2), d = 2 * (e % (HD / 2));
            const float2 v = *reinterpret_cast<const float2 *>(cpart + C::cp_index(h, d));
            if (p.direct_out) {
                const float gsum = ml_s[2 * h + 1];
                float *dst = p.out + ((size_t)it_lane * p.n_q + qh0 + h) * HD + d;
                dst[0] = gsum > 0.f ? v.x / gsum : 0.f;
                dst[1] = gsum > 0.f ? v.y / gsum : 0.f;
            } else {
                *reinterpret_cast<float2 *>(part_of(h, it_split) + 2 + d) = v;
            }
        }
        if (!p.direct_out && threadIdx.x < gvalid)
            *reinterpret_cast<float2 *>(part_of(threadIdx.x, it_split)) = make_float2(ml_s[2 * threadIdx.x], ml_s[2 * threadIdx.x + 1]);
    }
}

template <typename C, bool QUEUE>
int launch_as(lc_batch *b, const TqAttnParams &p, dim3 grid) {
    static lc_smem_optin optin;
    LC_CUDA_TRY(lc_ensure_smem(tq_attn_mma_kernel<C, QUEUE>, optin, b->ctx, C::SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(C::NT);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    LcPlain plain(b);
    if (b->ctx->pdl && !plain.serial) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    if (p.cluster_merge) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = p.n_splits;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        na++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    LC_LAUNCH_CHECKED(cudaLaunchKernelEx(&cfg, tq_attn_mma_kernel<C, QUEUE>, p));
    b->dispatch_count++;
    return LC_OK;
}

template <typename C>
int launch(lc_batch *b, const TqAttnParams &p, dim3 grid) {
    return p.queue_chunk != 0u ? launch_as<C, true>(b, p, grid) : launch_as<C, false>(b, p, grid);
}

template <int HD>
int launch_bits(lc_batch *b, const TqAttnParams &p, dim3 grid, uint32_t bits) {
    switch (bits) {
        case 2: return launch<AttnCfg<HD, 2>>(b, p, grid);
        case 3: return launch<AttnCfg<HD, 3>>(b, p, grid);
        default: return launch<AttnCfg<HD, 4>>(b, p, grid);
    }
}

}  // namespace

bool lc_tq_attn_mma_supported(uint32_t hd, uint32_t bits) { return (hd == 128 || hd == 256 || hd == 512) && bits >= 2 && bits <= 4; }

int lc_tq_attn_mma_launch(lc_batch *b, const TqAttnParams &p, dim3 grid, uint32_t hd, uint32_t bits) {
    switch (hd) {
        case 128: return launch_bits<128>(b, p, grid, bits);
        case 256: return launch_bits<256>(b, p, grid, bits);
        default: return launch_bits<512>(b, p, grid, bits);
    }
}

// (asked of one of the kernels that fill an SM's shared memory; the others that do differ in nothing that counts here)
void lc_cluster_capacity(const lc_ctx *ctx, uint32_t (&cap)[9]) {
    using C = AttnCfg<256, 2>;
    auto kern = tq_attn_mma_kernel<C, false>;
    cap[0] = 0;
    cap[1] = (uint32_t)ctx->sm_count;
    const bool ready = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) == cudaSuccess;
    for (uint32_t s = 2; s <= 8; s++) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(s);
        cfg.blockDim = dim3(C::NT);
        cfg.dynamicSmemBytes = C::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = s;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (!ready || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = ctx->sm_count * 3 / 4 / (int)s;
        }
        cap[s] = n < 1 ? 1u : (uint32_t)n;
    }
}
