// Shared declarations of the sm_100a MoE library: error plumbing, handle
// structs, launch prototypes of every kernel file.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../include/lmoe.h"

#define QK_K 256
#define Q4K_BYTES 144
#define Q6K_BYTES 210

// ---- error plumbing (thread-local message, status code) --------------------
lmoe_status lmoe_fail(lmoe_status code, const char *fmt, ...);
void lmoe_clear_error();

#define LMOE_CUDA(expr)                                                                            \
    do {                                                                                           \
        cudaError_t e__ = (expr);                                                                  \
        if (e__ != cudaSuccess)                                                                    \
            return lmoe_fail(LMOE_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__));      \
    } while (0)

// Kernels that follow one another in a call are launched with programmatic stream serialization: the next one's blocks may
// become resident while the last one still runs, and its launch latency (1 us each, ten kernels a call) is hidden.  Such a
// kernel begins with pdl_begin(): it waits until the kernel before it is complete and visible, and only then lets the one
// after it start, so that never more than two overlap.  Where there is nothing to wait for the two instructions do nothing.
// (70 tokens: 374 -> 364 us, 200: 446 -> 432; 130 tokens of a layer with 128 experts of 768: 181 -> 167; op by op, 3 tokens:
// 134 -> 118.)  The grouped products set up their barriers and tensor memory before they wait, and do not let the next kernel
// start early.  The two kernels that stream their results and the warp-per-row mat-vec are launched the plain way: overlapping
// those cost 2 to 4 % from 2048 tokens on, and up to half as much again.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
#endif

#define LMOE_LAUNCH_CHECK(name)                                                                    \
    do {                                                                                           \
        cudaError_t e__ = cudaGetLastError();                                                      \
        if (e__ != cudaSuccess)                                                                    \
            return lmoe_fail(LMOE_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e__)); \
    } while (0)

// ---- handles ----------------------------------------------------------------
struct lmoe_expert_stack {
    int32_t dtype;
    int64_t n_expert, n_out, k;
    const uint8_t *base; // device allocation (or caller's buffer for wrapped stacks)
    size_t base_off;     // first super-block = base + base_off
    size_t nbytes;       // bytes of super-blocks
    bool owned;
    int device;
    const uint8_t *blocks() const { return base + base_off; }
    int type_size() const { return dtype == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES; }
    int64_t row_bytes() const { return k / QK_K * type_size(); }
    int64_t expert_bytes() const { return n_out * row_bytes(); }
};

struct lmoe_layer {
    int64_t hidden, expert_ff, n_expert, top_k;
    float scale;
    int32_t norm;
    const float *router, *bias;
    const lmoe_expert_stack *gate, *up, *down, *sh_gate, *sh_up, *sh_down;
    // device words the fused decode kernel synchronises its CTAs through; zero between launches,
    // so one decode call at a time per layer
    uint32_t *sync;
    // guard of that rule: the stream and completion event of the latest decode call.  A call on a
    // different stream while the event is still pending is refused instead of corrupting `sync`.
    mutable std::mutex dec_mutex;
    mutable cudaEvent_t dec_event = nullptr;
    mutable cudaStream_t dec_stream = nullptr;
    mutable bool dec_pending = false;
    // Host-buffer decode calls: two device staging rows-buffers, filled by a copy stream of the layer's own, so that
    // the host-to-device copy of a call runs while the previous call's kernel does (created at the first such call).
    mutable std::mutex host_mutex;
    mutable float *host_x[2] = {nullptr, nullptr};
    mutable cudaStream_t host_copy_stream = nullptr;
    mutable cudaEvent_t host_copied[2] = {nullptr, nullptr}, host_slot_free[2] = {nullptr, nullptr};
    mutable int host_slot = 0;
    mutable bool host_failed = false;
};

static inline int lmoe_type_size(int32_t dtype) {
    return dtype == LMOE_Q4_K ? Q4K_BYTES : dtype == LMOE_Q6_K ? Q6K_BYTES : 0;
}

static inline size_t lmoe_align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---- kernel launchers (one per .cu file) -----------------------------------
// route.cu
cudaError_t launch_route_logits(const float *router, const float *x, int t, int hidden, int n_expert,
                                float *logits, cudaStream_t s);
cudaError_t launch_route_select(const float *logits, const float *bias, int t, int n_expert, int top_k,
                                float scale, int norm, uint32_t *ids, float *weights, cudaStream_t s, uint32_t *clear = nullptr);
// route_filter.cu
// Logits and selection in one, for long prompts: the same ids and weights.  `flag` is cleared first.
bool route_filter_available(int64_t hidden, int64_t n_expert, int64_t top_k);
size_t route_filter_bytes(int64_t t, int64_t hidden, int64_t n_expert);
cudaError_t launch_route_filter(const float *router, const float *bias, const float *x, int t, int hidden, int n_expert, int top_k, float scale, int norm,
                                void *scratch, uint32_t *ids, float *weights, uint32_t *flag, cudaStream_t s);
// mv_stream.cu
// Streamed Q6_K mat-vec: one activation row, all rows of the matrix.
bool mv_q6k_stream_available(int64_t n_out, int64_t k);
cudaError_t launch_mv_q6k_stream(const uint8_t *w, int n_out, int k, const float *x, float *out, cudaStream_t s);
// mv_id.cu
cudaError_t launch_mul_mv_id(int dtype, const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k,
                             const float *x, int t, int x_per_row, const uint32_t *ids, int top_k, float *out,
                             cudaStream_t s);
// mv_dense.cu
cudaError_t launch_mv_dense(int dtype, const uint8_t *w, int n_out, int k, const float *x, int64_t pairs, int x_per_row, const uint32_t *ids, int top_k,
                            float *out, cudaStream_t s);
// One product of launch_mul_mv_id_jobs: `pairs` = tokens times top_k; ids NULL = expert 0 for every pair.
constexpr int MV_JOBS = 4;
struct MvJob {
    const uint8_t *w;
    int64_t expert_bytes;
    int n_expert;
    const float *x;
    int x_per_row;
    const uint32_t *ids;
    int top_k, pairs;
    float *out;
};
// Products of the same type, row count and k that do not depend on one another.
cudaError_t launch_mul_mv_id_jobs(int dtype, const MvJob *job, int jobs, int n_out, int k, cudaStream_t s);
// glue.cu
// silu_mul and l2_rescale of rows of n values (a multiple of 256, at most LMOE_FFN_MM_MAX_FF), straight into the grouped GEMM's tile order as f16
// (row of the tile order pos[row], tiles of nt rows); a row that no list names (pos < 0) is a zero row of y instead.
cudaError_t launch_silu_rescale_tiles(const float *g, const float *u, const int32_t *pos, int64_t rows, int n, int nt, void *act, float *l2,
                                      float *y, int n_y, cudaStream_t s);
cudaError_t launch_silu_mul(const float *g, const float *u, int64_t n, float *out, cudaStream_t s);
cudaError_t launch_l2_rescale(const float *a, int64_t rows, int n, float *out, float *l2, cudaStream_t s);
cudaError_t launch_combine(const float *down, const float *col_l2, const float *w, int seq, int top_k,
                           int n_out, float *out, cudaStream_t s, const uint32_t *flag = nullptr);
cudaError_t launch_add_inplace(float *out, const float *b, int64_t n, cudaStream_t s);
cudaError_t launch_ep_localize_ids(const uint32_t *ids, int64_t n, uint32_t first, uint32_t count, uint32_t *out,
                                   cudaStream_t s);
cudaError_t launch_rms_norm(const float *x, const float *w, float eps, int64_t t, int hidden, float *out, cudaStream_t s);
cudaError_t launch_map0(const uint32_t *ids, int t, int top_k, int n_expert, uint32_t *tpe, int32_t *ids_map,
                        cudaStream_t s);
// codec.cu
cudaError_t launch_quantize(int dtype, const float *src, int64_t nblocks, uint8_t *dst, cudaStream_t s);
cudaError_t launch_dequantize(int dtype, const uint8_t *src, int64_t nblocks, float *dst, cudaStream_t s);
