// Routing of the quantized batched matmul C[m, n] = A[m, k] x W[n, k]^T, the
// stand-in for Kernels::matmul_nt_q4_0_into / matmul_nt_tq2_0_into
// (local-metal/src/kernels.rs:6459-6563).  The reference picks between four
// Metal kernels by m (batchm <= 4, smallm <= 8, simdgroup MMA, scalar tile); here
//   m <= 8, two groups of 64 rows per SM or more: the streaming kernel (qmatvec_mma.cu);
//   m <= 16: the small-batch kernel (qmatmul_sm.cu), but for wide Q4_0 outputs at short K;
//   TQ2_0, 16 < m <= 64: the tcgen05 decode kernel (qmatmul_tcd.cu);
//   Q4_0, f32 out, m > 8, 128 rows per SM or more: the vocabulary kernel (qmatmul_tcv.cu), 64 batch rows at a time;
//   other Q4_0, 16 < m <= 64: f32 out the register-direct kernels (qmatmul_mma.cu), f16 out those or the large-batch one, by
//     their estimates;
//   m > 64: the large-batch tcgen05 kernel (qmatmul_tcl.cu).
// The matvec entry points (lc_matvec_*, qmatvec.cu) take the first two as well.  What a kernel declines falls through to the
// next, and in the end to the CUDA-core kernels (qmatvec.cu).
// LOCAL_AI_MMA=0 forces the CUDA-core path for every m, as it forces the non-MMA
// kernels in the reference; LOCAL_CUDA_SMALL_M=n keeps TQ2_0 of up to n rows on it (or the streaming kernel); LOCAL_CUDA_DECODE_TC=0 /
// LOCAL_CUDA_DECODE_MMA=0 switch the tcgen05 and the mma.sync kernels of m <= 64 off (with both off, 8 < m <= 64 runs on
// qmatmul_tcl.cu as well).
#include <stdlib.h>
#include "lc_internal.h"

int lc_qgemm_cuda_core(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input,
                       const lc_buf *weight, lc_buf *output, uint32_t m, uint32_t kk, uint32_t n);
int lc_check_qargs(int fmt, const char *name, lc_kernels *k, lc_batch *b, const lc_buf *w, const lc_buf *x,
                   const lc_buf *out, uint32_t m, uint32_t kk, uint32_t n, size_t out_elem);
// qmatmul_tcl.cu: large-batch tcgen05 kernel, up to three matrices on the same activations; returns LC_OK when it launched, or
// a negative value when the shape is outside what it covers (caller falls through).
int lc_qgemm_tcl_launch(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                        lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk);
uint64_t lc_qgemm_tcl_estimate(const lc_kernels *k, uint32_t m, uint32_t kk, uint32_t n);   // ns, one Q4_0 matrix, 16 < m <= 64

// qmatmul_mma.cu: same contract, for 8 < m <= 64.
uint64_t lc_qgemm_mma_estimate(const lc_kernels *k, uint32_t m, uint32_t kk, uint32_t n);   // as above
int lc_qgemm_mma_grouped(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int ng,
                         const lc_buf *const *weights, lc_buf *const *outputs, const uint32_t *ns, uint32_t m,
                         uint32_t kk);

// qmatmul_tcd.cu: tcgen05 decode matmul (TQ2_0, f16 out, m <= 64); same return contract.
int lc_qgemm_tcd_launch(lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                        lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk, bool geglu);

// qmatmul_sm.cu: small-batch tensor-core kernel (both formats, f16 and f32 out, m <= 16); same return contract.
int lc_qgemm_sm_launch(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                       lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk, bool geglu);
int lc_qgemv_mma_stream(int fmt, bool f32out, lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                        lc_buf *output, uint32_t m, uint32_t kk, uint32_t n);
constexpr uint32_t SM_MAX_M = 16;
static bool small_batch_ok(const lc_kernels *k, int fmt, uint32_t m) {
    return k->mma && k->decode_mma && m <= SM_MAX_M && (fmt == 0 || (k->decode_tc && m > k->small_m));
}

// qmatmul_tcv.cu: persistent tcgen05 kernel for very tall Q4_0 matrices (the vocabulary projection), f32 out, m <= 64;
// same return contract.
int lc_qgemm_tcv_launch(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight, lc_buf *output, uint32_t m,
                        uint32_t kk, uint32_t n);

static int route(int fmt, bool f32out, const char *name, lc_kernels *k, lc_batch *b, const lc_buf *input,
                 const lc_buf *weight, lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    int st = lc_check_qargs(fmt, name, k, b, weight, input, output, m, kk, n, f32out ? 4 : 2);
    if (st != LC_OK) return st;
    if (n == 0) return LC_OK;
    const lc_buf *ws[1] = {weight};
    lc_buf *os[1] = {output};
    const uint32_t ns[1] = {n};
    if (small_batch_ok(k, fmt, m)) {
        st = m <= 8 ? lc_qgemv_mma_stream(fmt, f32out, k, b, input, weight, output, m, kk, n) : -1;
        if (st >= 0) return st;
        if (!(k->vocab_tc && fmt == 0 && f32out && m > 8 && n >= 128u * (uint32_t)k->ctx->sm_count)) {   // (the vocabulary kernel's shapes)
            st = lc_qgemm_sm_launch(fmt, f32out, k, b, input, 1, ws, os, ns, m, kk, false);
            if (st >= 0) return st;
        }
    }
    if (k->mma && k->decode_tc && fmt == 1 && !f32out && m > k->small_m && m <= 64) {
        st = lc_qgemm_tcd_launch(k, b, input, 1, ws, os, ns, m, kk, false);
        if (st >= 0) return st;
    }
    if (k->mma && k->vocab_tc && fmt == 0 && f32out && m > 8) {
        // The persistent vocabulary kernel takes 64 batch rows per launch; larger batches go through it in chunks.
        // Each chunk streams the table once, and still 262144 x 1536 at 128 / 256 / 512 rows takes 238 / 474 / 970 us
        // against 762 / 1510 / 2999 us for the large-batch kernel's predecessor; the present one is level with the chunks (267 us
        // against 265 at 128 rows).
        bool covered = m <= 4096;
        for (uint32_t m0 = 0; m0 < m && covered; m0 += 64) {
            const uint32_t mc = m - m0 < 64 ? m - m0 : 64;
            lc_buf in_v = *input, out_v = *output;
            in_v.dptr = (char *)input->dptr + (size_t)m0 * kk * 2;
            in_v.bytes = input->bytes - (size_t)m0 * kk * 2;
            in_v.owned = false;
            out_v.dptr = (char *)output->dptr + (size_t)m0 * n * 4;
            out_v.bytes = output->bytes - (size_t)m0 * n * 4;
            out_v.owned = false;
            st = lc_qgemm_tcv_launch(k, b, &in_v, weight, &out_v, mc, kk, n);
            if (st > 0) return st;
            if (st < 0) {
                if (m0 != 0) return lc_fail(LC_ERR_INVALID_ARGUMENT, "%s: vocabulary kernel declined chunk %u after accepting the first", name, m0 / 64);
                covered = false;
            }
        }
        if (covered) return LC_OK;
    }
    if (k->mma && m > 8) {
        if (m <= 64) {
            // Q4_0 from 17 rows: the large-batch kernel, or for a tall matrix at short K whichever kernel's estimate is less (large-batch
            // against register-direct: 24 x 40000 x 256 11.2 us and 9.0; 24 x 40000 x 512 14.2 and 13.6; 24 x 24000 x 512 9.3 and 10.8; 48 x 40000 x 256
            // 11.9 and 16.5; 48 x 71000 x 512 21.1 and 30.4; 64 x 150000 x 256 35.3 and 32.3).
            // f32 outputs keep the other: its sums, 32 k at a time, are within 1e-7 of 64 bits, the tcgen05 accumulators' within 1e-6.  (An f16
            // output hides that: over 56 shapes 2.07e-4 off 64 bits from either, their ratio 1.00002 in the mean and 1.00025 at most.)
            const bool choose = k->decode_tc && fmt == 0 && m > SM_MAX_M && !f32out;
            if (k->decode_mma && (!choose || lc_qgemm_mma_estimate(k, m, kk, n) < lc_qgemm_tcl_estimate(k, m, kk, n))) {
                st = lc_qgemm_mma_grouped(fmt, f32out, k, b, input, 1, ws, os, ns, m, kk);
                if (st >= 0) return st;
            }
        }
        st = lc_qgemm_tcl_launch(fmt, f32out, k, b, input, 1, ws, os, ns, m, kk);
        if (st >= 0) return st;
    }
    return lc_qgemm_cuda_core(fmt, f32out, k, b, input, weight, output, m, kk, n);
}

// Several TQ2_0 projections of the same activations (Q/K/V; gate/up) as one launch when the tensor-core
// path applies, else one after the other.
int lc_matmul_nt_tq2_0_grouped(lc_kernels *k, lc_batch *b, const lc_buf *input, int ng, const lc_buf *const *weights,
                               lc_buf *const *outputs, const uint32_t *ns, uint32_t m, uint32_t kk) {
    for (int g = 0; g < ng; g++) {
        int st = lc_check_qargs(1, "matmul_nt_tq2_0", k, b, weights[g], input, outputs[g], m, kk, ns[g], 2);
        if (st != LC_OK) return st;
    }
    if (small_batch_ok(k, 1, m)) {
        const int st = lc_qgemm_sm_launch(1, false, k, b, input, ng, weights, outputs, ns, m, kk, false);
        if (st >= 0) return st;
    }
    if (k->mma && k->decode_tc && m > k->small_m && m <= 64) {
        const int st = lc_qgemm_tcd_launch(k, b, input, ng, weights, outputs, ns, m, kk, false);
        if (st >= 0) return st;
    }
    if (k->mma && m > 8) {
        int st = -1;
        if (k->decode_mma && m <= 64) st = lc_qgemm_mma_grouped(1, false, k, b, input, ng, weights, outputs, ns, m, kk);
        if (st < 0) st = lc_qgemm_tcl_launch(1, false, k, b, input, ng, weights, outputs, ns, m, kk);
        if (st >= 0) return st;
    }
    for (int g = 0; g < ng; g++) {
        int st = lc_qgemm_cuda_core(1, false, k, b, input, weights[g], outputs[g], m, kk, ns[g]);
        if (st != LC_OK) return st;
    }
    return LC_OK;
}

int lc_qgemm_mma_geglu(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *w_gate, const lc_buf *w_up,
                       lc_buf *output, uint32_t m, uint32_t kk, uint32_t n);

extern "C" {

// The GeGLU half of the feed-forward block, gelu_tanh(x W_gate^T) * (x W_up^T) (local-engine/src/layer.rs:825-838):
// one launch on the decode path (8 < m <= 64), else the two projections into `gate_tmp` / `up_tmp` followed by
// gelu_mul.  `output` may alias `gate_tmp`.
int lc_matmul_nt_tq2_0_geglu_into(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *w_gate,
                                  const lc_buf *w_up, lc_buf *gate_tmp, lc_buf *up_tmp, lc_buf *output, uint32_t m,
                                  uint32_t kk, uint32_t n) {
    if (!gate_tmp || !up_tmp) return lc_fail(LC_ERR_INVALID_ARGUMENT, "matmul_nt_tq2_0_geglu: NULL argument");
    int st = lc_check_qargs(1, "matmul_nt_tq2_0_geglu", k, b, w_gate, input, output, m, kk, n, 2);
    if (st == LC_OK) st = lc_check_qargs(1, "matmul_nt_tq2_0_geglu", k, b, w_up, input, up_tmp, m, kk, n, 2);
    if (st == LC_OK) st = lc_check_qargs(1, "matmul_nt_tq2_0_geglu", k, b, w_gate, input, gate_tmp, m, kk, n, 2);
    if (st != LC_OK) return st;
    if (n == 0 || m == 0) return LC_OK;
    static const bool fused_ok = []() { const char *e = getenv("LOCAL_CUDA_GEGLU_FUSED"); return !(e && e[0] == '0'); }();
    if (fused_ok && k->mma && m > k->small_m && m <= 64) {
        if (k->decode_tc) {
            const lc_buf *ws[2] = {w_gate, w_up};
            lc_buf *os[2] = {output, output};
            const uint32_t ns[2] = {n, n};
            if (small_batch_ok(k, 1, m)) {
                st = lc_qgemm_sm_launch(1, false, k, b, input, 2, ws, os, ns, m, kk, true);
                if (st >= 0) return st;
            }
            st = lc_qgemm_tcd_launch(k, b, input, 2, ws, os, ns, m, kk, true);
            if (st >= 0) return st;
        }
        if (k->decode_mma && m > 8) {
            st = lc_qgemm_mma_geglu(k, b, input, w_gate, w_up, output, m, kk, n);
            if (st >= 0) return st;
        }
    }
    const lc_buf *ws[2] = {w_gate, w_up};
    lc_buf *os[2] = {gate_tmp, up_tmp};
    const uint32_t ns[2] = {n, n};
    st = lc_matmul_nt_tq2_0_grouped(k, b, input, 2, ws, os, ns, m, kk);
    if (st != LC_OK) return st;
    return lc_gelu_mul_into(k, b, gate_tmp, up_tmp, output, m * n);
}

int lc_matmul_nt_q4_0_into(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                           lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    return route(0, false, "matmul_nt_q4_0", k, b, input, weight, output, m, kk, n);
}

int lc_matmul_nt_tq2_0_into(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                            lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    return route(1, false, "matmul_nt_tq2_0", k, b, input, weight, output, m, kk, n);
}

int lc_matmul_nt_q4_0_f32out_into(lc_kernels *k, lc_batch *b, const lc_buf *input, const lc_buf *weight,
                                  lc_buf *output, uint32_t m, uint32_t kk, uint32_t n) {
    return route(0, true, "matmul_nt_q4_0_f32out", k, b, input, weight, output, m, kk, n);
}

}  // extern "C"
