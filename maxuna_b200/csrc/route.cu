// Stand-alone routing kernels: router logits (bit-specified f32 reduction) and
// the sigmoid / bias / ordered top-k / normalise step.
// Reference: `route_logits` and `route_from_logits`, src/moe.rs:84-119.
#include "common.cuh"
#include "route_math.cuh"
#include "route_tile.cuh"

namespace {

constexpr int ROUTE_WARPS = 8;

// grid (ceil(n_expert / WARPS), ceil(t / TT)); one warp per expert row,
// TT tokens per pass so the router row is read once per token tile.
template <int TT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
route_logits_kernel(const float *__restrict__ router, const float *__restrict__ x, int t, int hidden,
                    int n_expert, float *__restrict__ logits) {
    pdl_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = blockIdx.x * WARPS + warp;
    const int t0 = blockIdx.y * TT;
    if (e >= n_expert) return;
    constexpr int UNROLL = TT == 1 ? 12 : 6; // loads in flight: the kernel is their latency
    const float *w = router + (size_t)e * hidden;
    float acc[TT][4];
#pragma unroll
    for (int i = 0; i < TT; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;

    if ((hidden & 3) == 0) {
        const int full = hidden / 128; // passes where every lane has a full float4
#pragma unroll UNROLL
        for (int j = 0; j < full; j++) {
            const float4 wv = __ldg(reinterpret_cast<const float4 *>(w + 128 * j + 4 * lane));
#pragma unroll
            for (int i = 0; i < TT; i++) {
                if (t0 + i < t) {
                    const float4 xv =
                        __ldg(reinterpret_cast<const float4 *>(x + (size_t)(t0 + i) * hidden + 128 * j + 4 * lane));
                    acc[i][0] = __fmaf_rn(xv.x, wv.x, acc[i][0]);
                    acc[i][1] = __fmaf_rn(xv.y, wv.y, acc[i][1]);
                    acc[i][2] = __fmaf_rn(xv.z, wv.z, acc[i][2]);
                    acc[i][3] = __fmaf_rn(xv.w, wv.w, acc[i][3]);
                }
            }
        }
        const int base = 128 * full + 4 * lane; // ragged last pass (hidden % 128 != 0)
        if (base < hidden) {
            const float4 wv = __ldg(reinterpret_cast<const float4 *>(w + base));
#pragma unroll
            for (int i = 0; i < TT; i++) {
                if (t0 + i < t) {
                    const float4 xv = __ldg(reinterpret_cast<const float4 *>(x + (size_t)(t0 + i) * hidden + base));
                    acc[i][0] = __fmaf_rn(xv.x, wv.x, acc[i][0]);
                    acc[i][1] = __fmaf_rn(xv.y, wv.y, acc[i][1]);
                    acc[i][2] = __fmaf_rn(xv.z, wv.z, acc[i][2]);
                    acc[i][3] = __fmaf_rn(xv.w, wv.w, acc[i][3]);
                }
            }
        }
    } else {
        for (int j = 0; 128 * j < hidden; j++) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int idx = 128 * j + 4 * lane + c;
                if (idx < hidden) {
                    const float wv = w[idx];
#pragma unroll
                    for (int i = 0; i < TT; i++)
                        if (t0 + i < t) acc[i][c] = __fmaf_rn(x[(size_t)(t0 + i) * hidden + idx], wv, acc[i][c]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TT; i++) {
        const float v = lmoe_router_fold(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (lane == 0 && t0 + i < t) logits[(size_t)(t0 + i) * n_expert + e] = v;
    }
}

// hidden a multiple of 512 (route_tile.cuh).  grid (token tiles, shares of the experts)
template <int T>
__global__ void __launch_bounds__(RT_THREADS, 1)
route_logits_tiled_kernel(const float *__restrict__ router, const float *__restrict__ x, int t, int hidden, int n_expert,
                          int experts_per_block, float *__restrict__ logits) {
    pdl_begin();
    extern __shared__ __align__(16) uint8_t rt_smem[];
    const int t0 = blockIdx.x * T;
    route_tile<T>(router, [&](int tok) { return x + (size_t)(t0 + tok) * hidden; }, min(T, t - t0), hidden, n_expert, blockIdx.y * experts_per_block,
                  min(n_expert, (int)(blockIdx.y + 1) * experts_per_block), rt_smem, logits + (size_t)t0 * n_expert);
}

// One warp per token, up to 32 * PER experts in its registers.  (Rounds of a scan of shared memory and ten dependent shuffles
// were a chain of latencies: logits and selection of 3 tokens, 256 experts 15.2 -> 8.1 us, 64 33.6 -> 19.2, 512 40.8 -> 34.4.)
// clear: four words to set to zero (a call's device flag, which otherwise takes a launch of its own), or NULL.
template <int PER>
__global__ void __launch_bounds__(ROUTE_WARPS * 32)
route_select_kernel(const float *__restrict__ logits, const float *__restrict__ bias, int t, int n_expert,
                    int top_k, float scale, int norm, uint32_t *__restrict__ ids, float *__restrict__ weights, uint32_t *__restrict__ clear) {
    pdl_begin();
    if (clear && blockIdx.x == 0 && threadIdx.x < 4) clear[threadIdx.x] = 0u;
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int token = blockIdx.x * ROUTE_WARPS + warp;
    if (token >= t) return;
    const float *lg = logits + (size_t)token * n_expert;
    float *probs = smem + (size_t)warp * n_expert;
    uint32_t key[PER];
    float v[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) v[j] = lane + 32 * j < n_expert ? __ldg(lg + lane + 32 * j) : 0.f;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int e = lane + 32 * j;
        key[j] = 0u;
        if (e < n_expert) {
            const float p = lmoe_sigmoid_fixed(v[j]);
            probs[e] = p;
            key[j] = lmoe_score_key(bias ? __fadd_rn(p, __ldg(bias + e)) : p);
        }
    }
    __syncwarp();
    lmoe_warp_select_keys<PER>(key, probs, top_k, scale, norm, ids + (size_t)token * top_k, weights + (size_t)token * top_k, lane);
}

} // namespace

cudaError_t launch_route_logits(const float *router, const float *x, int t, int hidden, int n_expert,
                                float *logits, cudaStream_t s) {
    if (t == 0) return cudaSuccess;
    constexpr int LOGIT_WARPS = 2; // few blocks are what a small batch has: 256 experts on 128 SMs instead of 32
    const unsigned gx = (unsigned)((n_expert + LOGIT_WARPS - 1) / LOGIT_WARPS);
    static int sms_of[64] = {0}; // per device: SM count, and the shared-memory opt-in done once
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!sms_of[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
        cudaFuncSetAttribute(route_logits_tiled_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        cudaFuncSetAttribute(route_logits_tiled_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        sms_of[dev] = n;
    }
    // A warp per expert row while its blocks are few, up to five an SM; beyond, their trips to the L2 cache take longer than a
    // register-tiled pass, whose time is the same for any small batch (256 experts, 16 / 24 / 64 tokens: 11.0 / 12.8 / 19.1 us
    // against 12.4 / 12.5 / 12.8; 64 experts of 4096, 64 tokens: 10.2 against 13.3).
    // The tile is padded to 16 experts: up to eight are better off untiled until the tokens are many (8 experts of 4096, 1024 /
    // 2048 / 4096 tokens: 16.9 / 26.9 / 48 us tiled, 11.1 / 19.4 / 36 so).
    const bool many = (int64_t)gx * ((t + 3) / 4) > 5 * sms_of[dev] && (n_expert > 8 || t > 4096);
    if (many && hidden % (128 * RT_AHEAD) == 0 && 8 * hidden * 4 + RT_FOLD <= 227 * 1024) {
        // One block per SM at a time: 16 tokens and 16 experts a pass where the rows fit (hidden <= 3072), or 8 tokens and 32
        // experts, in the same time.  The experts are split over blocks until the device is covered, and further where that
        // fills the last wave better; a block repeats the staging of its tokens, which for 16 costs about a pass.  Of equal
        // choices the one that reads the router less (130 tokens 17.0 us with 8 and 18.3 with 16, selection included).
        int nt = 0, pass = 0, ppb = 0;
        int64_t best = INT64_MAX;
        for (int n = 16; n >= 8; n -= 8) {
            if (n * hidden * 4 + RT_FOLD > 227 * 1024) continue;
            const int tiles = (t + n - 1) / n, ex = 256 / n, passes = (n_expert + ex - 1) / ex;
            for (int p = passes; p >= 1; p--) {
                const int64_t blocks = (int64_t)tiles * ((passes + p - 1) / p);
                const int64_t cost = (blocks + sms_of[dev] - 1) / sms_of[dev] * (2 * p + n / 8);
                if (cost < best) best = cost, nt = n, pass = ex, ppb = p;
            }
        }
        const dim3 grid((unsigned)((t + nt - 1) / nt), (unsigned)((n_expert + pass * ppb - 1) / (pass * ppb)));
        const int smem = nt * hidden * 4 + RT_FOLD;
        if (nt == 16)
            launch_pdl(route_logits_tiled_kernel<16>, grid, RT_THREADS, smem, s, router, x, t, hidden, n_expert, ppb * pass, logits);
        else
            launch_pdl(route_logits_tiled_kernel<8>, grid, RT_THREADS, smem, s, router, x, t, hidden, n_expert, ppb * pass, logits);
    } else if (t <= 2) {
        launch_pdl(route_logits_kernel<1, LOGIT_WARPS>, dim3(gx, t), LOGIT_WARPS * 32, 0, s, router, x, t, hidden, n_expert, logits);
    } else {
        // Rows of two or three steps are mostly fold: in very large numbers twice the warps a block, and the plain launch, which
        // spreads them evenly (hidden 256, 256 experts, 2048 / 16384 tokens 73 / 563 us as below, 51 / 351 so).
        const bool short_rows = hidden % 4 == 0 && hidden <= 384 && (int64_t)gx * ((t + 3) / 4) > 100 * (int64_t)sms_of[dev];
        constexpr int TOKENS = 65535 * 4; // grid.y is limited to 65535
        for (int t0 = 0; t0 < t; t0 += TOKENS) {
            const int n = t - t0 < TOKENS ? t - t0 : TOKENS;
            const float *xs = x + (size_t)t0 * hidden;
            float *ls = logits + (size_t)t0 * n_expert;
            if (short_rows)
                route_logits_kernel<4, 4><<<dim3((unsigned)((n_expert + 3) / 4), (n + 3) / 4), 128, 0, s>>>(router, xs, n, hidden, n_expert, ls);
            else
                launch_pdl(route_logits_kernel<4, LOGIT_WARPS>, dim3(gx, (n + 3) / 4), LOGIT_WARPS * 32, 0, s, router, xs, n, hidden, n_expert, ls);
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_route_select(const float *logits, const float *bias, int t, int n_expert, int top_k,
                                float scale, int norm, uint32_t *ids, float *weights, cudaStream_t s, uint32_t *clear) {
    if (t == 0) return cudaSuccess;
    const size_t smem = (size_t)ROUTE_WARPS * n_expert * sizeof(float);
    const unsigned grid = (unsigned)((t + ROUTE_WARPS - 1) / ROUTE_WARPS);
    if (n_expert > 512) return cudaErrorInvalidValue; // every entry point has refused it
    // a round rescans the lane's scores: no more of them than needed
    launch_pdl(n_expert <= 128 ? route_select_kernel<4> : (n_expert <= 256 ? route_select_kernel<8> : route_select_kernel<16>), grid,
               ROUTE_WARPS * 32, smem, s, logits, bias, t, n_expert, top_k, scale, norm, ids, weights, clear);
    return cudaGetLastError();
}

// ---- routing without any allocation -------------------------------------------------------
// Some hosts of this library may not allocate device memory at the moment they route: an engine
// whose buffer pool owns the whole device and hands nothing to plugins, a serving loop running
// under a frozen memory budget, or code that is between cudaStreamBeginCapture and EndCapture.
// For them the logits scratch of `lmoe_route` lives in this fixed array instead of a caller
// workspace.  Every GPU that loads the library carries the array until the process exits.
#define LMOE_ROUTE_NOALLOC_MAX_LOGITS (64 * 512) /* t * n_expert floats, 128 KB */
static __device__ __align__(256) float g_route_noalloc_logits[LMOE_ROUTE_NOALLOC_MAX_LOGITS];

extern "C" lmoe_status lmoe_route_noalloc(const float *router, const float *bias, const float *x, int64_t t,
                                          int64_t hidden, int64_t n_expert, int64_t top_k, float scale, int32_t norm,
                                          uint32_t *ids_out, float *weights_out, void *stream) {
    lmoe_clear_error();
    if (t < 0 || n_expert < 1 || n_expert > 512 || top_k < 1 || top_k > 32 || top_k > n_expert)
        return lmoe_fail(LMOE_ERR_INVALID, "route_noalloc: t >= 0, n_expert in [1, 512], top_k in [1, min(32, n_expert)] required");
    if (hidden < 1 || hidden > (1 << 20)) return lmoe_fail(LMOE_ERR_INVALID, "hidden (%lld) out of range", (long long)hidden);
    // t is bounded before the product is formed, so the comparison below cannot wrap around
    if (t > LMOE_ROUTE_NOALLOC_MAX_LOGITS || t * n_expert > LMOE_ROUTE_NOALLOC_MAX_LOGITS)
        return lmoe_fail(LMOE_ERR_INVALID,
                         "route_noalloc: t * n_expert = %lld exceeds the built-in scratch of %d logits; use lmoe_route with a workspace",
                         t > LMOE_ROUTE_NOALLOC_MAX_LOGITS ? (long long)t : (long long)(t * n_expert), LMOE_ROUTE_NOALLOC_MAX_LOGITS);
    if (!router || !x || !ids_out || !weights_out) return lmoe_fail(LMOE_ERR_INVALID, "router/x/ids_out/weights_out is NULL");
    if (hidden % 4 == 0 && (((uintptr_t)router | (uintptr_t)x) & 15u))
        return lmoe_fail(LMOE_ERR_INVALID, "router and x must be 16-byte aligned");
    // In host code the array's name is only a stand-in; the kernels need its device address, which
    // differs per GPU.  It is looked up once per device, with that device current.
    static float *dev_ptr[64] = {nullptr};
    int dev = 0;
    LMOE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "device ordinal %d not supported", dev);
    if (!dev_ptr[dev]) {
        float *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void **)&p, g_route_noalloc_logits);
        if (e != cudaSuccess || !p)
            return lmoe_fail(LMOE_ERR_CUDA, "cudaGetSymbolAddress(route scratch) failed: %s", cudaGetErrorString(e));
        dev_ptr[dev] = p;
    }
    float *logits = dev_ptr[dev];
    // nothing has to start at zero: every logit a launch reads was written by the same call
    LMOE_CUDA(launch_route_logits(router, x, (int)t, (int)hidden, (int)n_expert, logits, (cudaStream_t)stream));
    LMOE_CUDA(launch_route_select(logits, bias, (int)t, (int)n_expert, (int)top_k, scale, norm, ids_out, weights_out,
                                  (cudaStream_t)stream));
    return LMOE_OK;
}
