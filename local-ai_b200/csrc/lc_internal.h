// Internal definitions shared by the translation units of liblocal_cuda.so.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/local_cuda.h"

// Which of a context's launches may run beside each other (LcOrder below).
struct lc_range {
    uintptr_t lo, hi;
};
struct lc_overlap {
    std::mutex mu;           // held from the decision about a launch until it is enqueued
    bool beside = false;     // the last launch runs beside others
    bool brief = false;      // the last launch recorded here takes the host longer than the GPU
    int state = 0;           // 0: nothing known, 1: `reads` / `writes` are the last launch's, 2: those of every launch that may be running
    int n_reads = 0, n_writes = 0;
    lc_range reads[192], writes[96];   // (when they are full the run starts anew)
    lc_range read_span = {}, write_span = {};   // what the lists span together
};

struct lc_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int sm_count = 0;
    size_t smem_optin = 0;
    size_t l2_bytes = 0;
    size_t total_mem = 0;
    bool pdl = true;  // launch kernels with programmatic stream serialization (LOCAL_CUDA_PDL=0 disables)
    // Launches whose buffers do not meet may overlap.  LOCAL_CUDA_OVERLAP=0 disables, and so does handing out the stream: work that
    // others put there is not seen here (lc_ctx_set_overlap).
    bool overlap_wanted = true;
    mutable std::atomic<bool> side_by_side{true};
    lc_overlap overlap;
};

struct lc_buf {
    lc_ctx *ctx = nullptr;
    void *dptr = nullptr;
    size_t bytes = 0;
    bool owned = false;
};

struct lc_batch {
    lc_ctx *ctx = nullptr;
    cudaStream_t stream = nullptr;
    uint32_t dispatch_count = 0;
    uint32_t last_order = 0;   // LcOrder::flags of the last launch, 0 where it declares nothing
    bool capturing = false;
};

struct lc_pending {
    int device = 0;   // not the context: a pending batch may outlive it
    cudaEvent_t ev = nullptr;
};

struct lc_graph {
    lc_ctx *ctx = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

struct lc_kernels {
    lc_ctx *ctx = nullptr;
    // Routing switches, read once like the reference's OnceLock-cached env flags.
    bool batchm = true;  // LOCAL_AI_BATCHM: register-resident small-M path
    bool smallm = true;  // LOCAL_AI_SMALLM
    bool mma = true;     // LOCAL_AI_MMA: tensor-core path for larger M
    bool decode_tc = true;   // LOCAL_CUDA_DECODE_TC: tcgen05 kernels at M <= 64 (TQ2_0 above small_m, Q4_0 from 17 rows), small-batch kernel for TQ2_0
    uint32_t small_m = 0;    // LOCAL_CUDA_SMALL_M (0..8): TQ2_0 matmuls of up to this many rows keep the CUDA-core kernel
    bool vocab_tc = true;    // LOCAL_CUDA_VOCAB_TC: persistent tcgen05 kernel for very tall Q4_0 matrices, f32 out, M <= 64
    bool decode_mma = true;  // LOCAL_CUDA_DECODE_MMA: mma.sync kernels at M <= 64 (0: tcgen05 or CUDA cores there too)
    int kv_norm_mode = 0;  // LOCAL_CUDA_TQ_NORM: 0 sequential (Rust codec order), 1 tree (Metal order)
    // Library-owned scratch for split-K partials (grown outside graph capture).
    void *scratch = nullptr;
    size_t scratch_bytes = 0;
    unsigned int *counters = nullptr;  // per-(lane,head) arrival counters, zero between launches
    size_t counters_len = 0;
    std::vector<void *> retired;  // outgrown scratch / counter blocks: graphs recorded earlier still point at them
    int *dev_status = nullptr;  // device-side error word (bounded waits report here)
    // Clusters of s CTAs, an SM each, that the device runs at once (lc_cluster_capacity).  A cluster needs all its SMs in one
    // GPC, so this is well below SMs / s: 74 pairs, but 45 triples, 33 fours and 15 eights on 148 SMs.  A launch of one more
    // runs a second wave and takes twice as long.
    uint32_t cluster_cap[9] = {0};
    // LOCAL_CUDA_TEST_WAIT_EXPIRY=1 (read at creation): the barrier waits of the matmuls (not of the streaming matvec) and of the
    // prefill attention kernel use a short limit and wait for an arrival that never comes, so the expiry path (status word, early
    // exit, TMEM release) can be exercised on purpose.
    bool test_wait_expiry = false;
    // LOCAL_CUDA_TEST_MAP_REFUSED=1 (read at creation): tensor maps over weights are as if the driver refused them, so that the copies
    // that serve without one can be exercised.
    bool test_map_refused = false;
};

// Values of the device-side status word (lc_kernels::dev_status).
constexpr int LC_DEV_STATUS_WAIT_EXPIRED = 1;      // a bounded barrier wait ran out (large-batch matmul, prefill attention, streaming matvec)
constexpr int LC_DEV_STATUS_WAIT_EXPIRED_TCD = 2;  // the same in the small-batch, decode and vocabulary matmuls
constexpr int LC_DEV_STATUS_POSITION = 3;          // a device-resident position pointed past its lane's pool rows

// Record a failure for lc_last_error() and return `code`.
int lc_fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
void lc_clear_error();

#define LC_CUDA_TRY(expr)                                                              \
    do {                                                                               \
        cudaError_t _e = (expr);                                                       \
        if (_e != cudaSuccess)                                                         \
            return lc_fail(LC_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(_e));      \
    } while (0)

#define LC_REQUIRE(cond, ...)                                          \
    do {                                                               \
        if (!(cond)) return lc_fail(LC_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
    } while (0)

#define LC_LAUNCH_CHECKED(expr)                                                        \
    do {                                                                               \
        cudaError_t _le = (expr);                                                      \
        if (_le != cudaSuccess)                                                        \
            return lc_fail(LC_ERR_CUDA, "launch: %s", cudaGetErrorString(_le));         \
    } while (0)

// After a kernel launch: surface launch-configuration errors as a status.
#define LC_CHECK_LAUNCH(name)                                                          \
    do {                                                                               \
        cudaError_t _e = cudaGetLastError();                                           \
        if (_e != cudaSuccess)                                                         \
            return lc_fail(LC_ERR_CUDA, "launch %s: %s", name, cudaGetErrorString(_e)); \
    } while (0)

// Every kernel of this library is launched through lc_launch so that it can start while its
// predecessor on the stream is still draining (programmatic dependent launch): a kernel calls
// lc_pdl_trigger() at its top — its successors may then be scheduled — and lc_pdl_wait() before it
// first touches memory a predecessor may have written.  Work that does not depend on the predecessor
// (streaming constant weights towards the SM) goes before the wait.
// A launch that declares nothing ends a run of launches side by side (LcOrder below); it lives until its launch is enqueued.  `serial`: the
// launch has to start only when its predecessor is complete (several of a run may still be running, and a kernel fetches its
// constant operands ahead of its wait).
class LcPlain {
public:
    explicit LcPlain(lc_batch *b) : lock(b->ctx->overlap.mu) {
        lc_overlap &o = b->ctx->overlap;
        o.state = 0;
        b->last_order = 0;
        if (b->stream == b->ctx->stream) {   // (runs are that stream's)
            serial = o.beside;
            o.beside = false;
        }
    }
    bool serial = false;

private:
    std::lock_guard<std::mutex> lock;
};
// After work that is no launch of this library's kernels: what LcOrder knows is no longer all that may be running.  `foreign`: a kernel
// of another library, which may let its successors start early; copies, memsets and graphs are complete before a later launch starts.
static inline void lc_order_break(lc_ctx *ctx, bool foreign = false) {
    std::lock_guard<std::mutex> lock(ctx->overlap.mu);
    ctx->overlap.state = 0;
    if (!foreign) ctx->overlap.beside = false;
}
// `serial`: the launch starts only when its predecessor is complete.
template <typename... KArgs, typename... Args>
static inline cudaError_t lc_launch_as(bool serial, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, lc_batch *b,
                                       Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = b->ctx->pdl && !serial ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
static inline cudaError_t lc_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, lc_batch *b,
                                    Args &&...args) {
    LcPlain plain(b);
    return lc_launch_as(plain.serial, kern, grid, block, smem, b, static_cast<KArgs>(args)...);
}
// Launches of one stream run one after the other because the next may read what the last wrote.  Several projections of the same
// activations, or the same projection of several matrices, do not: a launch of a few microseconds then spends most of its time
// on latency that the next one's work could hide.  The matmul kernels declare the bytes that they read and write; where those of
// a new launch do not meet those of the launches it would run beside, it does not wait for them:
//   * the first such launch waits for its predecessor as ever, but lets its successors start only after that wait (LC_LATE_TRIGGER),
//     so whatever came before is complete when they run;
//   * the following ones start at once and wait for their predecessor at their end (LC_LATE_WAIT), so that a launch is complete only
//     when all before it are.  One that depends on any that may be running waits for the last as ever; so do launches that declare
//     nothing, which end the run and, because a kernel fetches its constant operands ahead of its wait, start only when the last launch
//     of a run is complete (`serial`).
// Whatever else the library puts on the stream ends the run, too (lc_order_break: copies, memsets, collectives, graphs, capture
// boundaries), and a program that takes the stream for work of its own has no runs at all (lc_ctx_stream).  Ranges are virtual addresses: memory mapped twice is not recognised.
// (35 matrices of 8192 x 1536 TQ2_0 times 16 rows took 225 us one after the
// other and take 98 side by side, 35 of Q4_0 6144 x 1536 times 40 rows 348 and 269, 35 of Q4_0 8192 x
// 1536 times one row 206 and 113.  `brief`: outside a capture the host takes longer to enqueue the launch than the GPU to run it, so there is
// nothing to hide, while launches side by side cost the host 0.05 to 0.1 us each, of which the look at the ranges is 0.015; two such launches
// start no run.  35 of 1024 x 512 TQ2_0 times one row 94.7 us one after the other, 101 side by side.)
constexpr uint32_t LC_LATE_TRIGGER = 1, LC_LATE_WAIT = 2;
class LcOrder {
public:
    LcOrder(lc_batch *b, const lc_buf *input, size_t in_bytes, int ng, const lc_buf *const *weights, const size_t *w_bytes,
            lc_buf *const *outputs, const size_t *out_bytes, bool brief = false);
    ~LcOrder();
    uint32_t flags = 0;      // for the kernel
    bool serial = false;     // for the launch
    bool launched = false;   // set by the caller once its one launch is enqueued

private:
    lc_ctx *ctx;
};
#ifdef __CUDACC__
__device__ __forceinline__ void lc_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void lc_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The same for kernels launched under an LcOrder: at their top, before their first dependent access, and at their end (any one CTA
// keeps the grid from completing).  ORDERED: flags are set; without them the kernel is one that knows none (reading them ahead of the
// trigger cost a decode step 0.3 to 1.1 %).
template <bool ORDERED>
__device__ __forceinline__ void lc_order_begin(uint32_t flags) {
    if (!ORDERED || !(flags & LC_LATE_TRIGGER)) lc_pdl_trigger();
}
template <bool ORDERED>
__device__ __forceinline__ void lc_order_wait(uint32_t flags) {
    if (!ORDERED || !(flags & LC_LATE_WAIT)) lc_pdl_wait();
    if (ORDERED && (flags & LC_LATE_TRIGGER)) lc_pdl_trigger();
}
template <bool ORDERED>
__device__ __forceinline__ void lc_order_end(uint32_t flags) {
    if (ORDERED && (flags & LC_LATE_WAIT) && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) lc_pdl_wait();
}

// Walsh-Hadamard transform (unnormalised) over d = 32 .. 512 elements held one per thread of a d-thread block;
// returns the thread's element of the result.  Butterflies run in ascending stride, lower = a + b, upper = a - b.
// The strides below 32 pair lanes of one warp and run as shuffles.  For the strides from 32 up every thread
// publishes its value once in `sh` and rebuilds the butterflies its result depends on from the d / 32 values it
// needs: the same additions on the same operands as stage-by-stage passes through shared memory, hence bit-identical
// to them, with one barrier in all instead of two per stage.  No thread may still be reading `sh` from earlier code
// when the block enters (callers that used it since their last barrier place one), and callers that reuse `sh`
// afterwards synchronise first.
struct lc_block_sync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
template <int P, typename Sync = lc_block_sync>
__device__ __forceinline__ float lc_fwht_cross_warp(float v, float *sh, unsigned t, Sync sync = {}) {
    sh[t] = v;
    sync();
    float a[P];
#pragma unroll
    for (int j = 0; j < P; j++) a[j] = sh[t ^ ((unsigned)j << 5)];
#pragma unroll
    for (int s = 0; (1 << s) < P; s++) {
        const bool upper = t & (32u << s);
#pragma unroll
        for (int j = 0; j < P; j += 2 << s) {
            const float self_v = a[j], other_v = a[j | (1 << s)];
            a[j] = upper ? __fsub_rn(other_v, self_v) : __fadd_rn(self_v, other_v);
        }
    }
    return a[0];
}
__device__ __forceinline__ float lc_fwht_value(float v, float *sh, unsigned d, unsigned t) {
#pragma unroll
    for (unsigned len = 1; len < 32; len <<= 1) {
        const float other_v = __shfl_xor_sync(0xffffffffu, v, len);
        v = (t & len) ? __fsub_rn(other_v, v) : __fadd_rn(v, other_v);
    }
    switch (d) {
        case 64: return lc_fwht_cross_warp<2>(v, sh, t);
        case 128: return lc_fwht_cross_warp<4>(v, sh, t);
        case 256: return lc_fwht_cross_warp<8>(v, sh, t);
        case 512: return lc_fwht_cross_warp<16>(v, sh, t);
        default: return v;   // d == 32
    }
}
#endif

// The opt-in to more than 48 KB of dynamic shared memory is a per-device attribute of a kernel.  One
// lc_smem_optin (a function-local static at each launch site, i.e. one per kernel instantiation) remembers
// the largest size already granted on each device, so every device a context is created on gets its own call.
constexpr int LC_MAX_DEVICES = 64;
struct lc_smem_optin {
    std::atomic<size_t> granted[LC_MAX_DEVICES];
};
template <typename Kern>
static inline cudaError_t lc_ensure_smem(Kern kern, lc_smem_optin &state, const lc_ctx *ctx, size_t smem) {
    if (smem <= 40 * 1024) return cudaSuccess;   // (48 KB less what a kernel may have of static shared memory)
    const int dev = ctx->device;
    if (dev >= 0 && dev < LC_MAX_DEVICES && state.granted[dev].load(std::memory_order_relaxed) >= smem) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && dev >= 0 && dev < LC_MAX_DEVICES) state.granted[dev].store(smem, std::memory_order_relaxed);
    return e;
}

static inline bool lc_aligned(const void *p, size_t a) { return ((uintptr_t)p & (a - 1)) == 0; }

void lc_cluster_capacity(const lc_ctx *ctx, uint32_t (&cap)[9]);   // attention_tq_mma.cu

// Grow the kernels object's split-K scratch (no-op when large enough). Fails
// during graph capture if growth would be needed.
int lc_reserve_scratch(lc_kernels *k, lc_batch *b, size_t bytes, size_t counters);

// Run `body(batch)` on a fresh batch and wait: the shape of the reference's
// ctx-taking dispatchers (e.g. kernels.rs:5711-5742).
template <typename F>
static inline int lc_run_and_wait(lc_ctx *ctx, F body) {
    lc_batch *b = nullptr;
    int st = lc_batch_begin(ctx, &b);
    if (st != LC_OK) return st;
    st = body(b);
    int st2 = lc_batch_commit_and_wait(b);
    return st != LC_OK ? st : st2;
}
