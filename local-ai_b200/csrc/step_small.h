// The layers of a decode step for few lanes in one launch (step_small.cu).
#pragma once
#include "lc_internal.h"

constexpr uint32_t LC_STEP_MAX_LANES = 4;      // (step_small.cu says why)
constexpr uint32_t LC_STEP_MAX_LAYERS = 64;    // the layers' pointers travel as a kernel parameter

struct LcStepLayer {
    const uint8_t *wq, *wk, *wv, *wo, *wgate, *wup, *wdown;   // TQ2_0
    const __half *attn_norm, *q_norm, *k_norm, *post_attn_norm, *ffn_norm, *post_ffn_norm;
    uint8_t *k_codes, *v_codes;
    __half *k_norms, *v_norms;
    uint32_t window, ring, lane_rows;
    uint32_t splits;                      // filled in by the launch: splits of a lane's keys, and where the layer's
    uint64_t mail;                        // exchange buffers start
};
// What the launch needs of a model; the caller fills in what stands before `status`.
struct LcStepParams {
    LcStepLayer layer[LC_STEP_MAX_LAYERS];
    int m, n_layers, hidden, inter, n_q, n_kv;
    const uint8_t *embed;                 // Q4_0 [vocab, hidden]
    const uint32_t *tokens, *positions;
    float embed_scale, eps, theta, softmax_scale;
    const __half *final_norm;
    const float *levels, *signs;
    __half *normed;                       // [m, hidden]: the final hidden rows
    uint8_t *mail;                        // lc_step_small_mail_bytes, for the exchange between the CTAs
    int *status;
    uint32_t wait_limit, never;           // never: 1 in the expiry self-test, nothing counts as arrived
    int off_b, off_u, off_rot, off_resid; // shared memory: second weight region, work space, rotations, residual rows;
    int off_red;                          // in the work space the sums
};
bool lc_step_small_supported(const lc_kernels *k, uint32_t hidden, uint32_t inter, uint32_t n_q, uint32_t n_kv, uint32_t head_dim,
                             uint32_t bits, uint32_t n_layers);
// for up to max_lanes lanes (at most LC_STEP_MAX_LANES); window and lane_rows of every layer as in LcStepLayer
size_t lc_step_small_mail_bytes(const lc_kernels *k, uint32_t hidden, uint32_t inter, uint32_t n_q, uint32_t n_kv, uint32_t n_layers,
                                uint32_t max_lanes, const uint32_t *window, const uint32_t *lane_rows);
// LC_OK after the launch, a positive status on error, -1 where the form does not fit (shared memory, alignment).
int lc_step_small_launch(lc_kernels *k, lc_batch *b, LcStepParams &p, uint32_t bits);
