// Stand-alone routing kernels: router logits (bit-specified f32 reduction) and
// the sigmoid / bias / ordered top-k / normalise step.
// Reference: `route_logits` and `route_from_logits`, src/moe.rs:84-119.
#include "common.cuh"
#include "route_math.cuh"

namespace {

constexpr int ROUTE_WARPS = 8;

// grid (ceil(n_expert / ROUTE_WARPS), ceil(t / TT)); one warp per expert row,
// TT tokens per pass so the router row is read once per token tile.
template <int TT>
__global__ void __launch_bounds__(ROUTE_WARPS * 32)
route_logits_kernel(const float *__restrict__ router, const float *__restrict__ x, int t, int hidden,
                    int n_expert, float *__restrict__ logits) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = blockIdx.x * ROUTE_WARPS + warp;
    const int t0 = blockIdx.y * TT;
    if (e >= n_expert) return;
    const float *w = router + (size_t)e * hidden;
    float acc[TT][4];
#pragma unroll
    for (int i = 0; i < TT; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;

    if ((hidden & 3) == 0) {
        const int full = hidden / 128; // passes where every lane has a full float4
#pragma unroll 4
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

// hidden a multiple of 128: a register-tiled product over the 128 partial chains of the specified order.
// A block stages 2 * NT tokens in shared memory and walks its share of the experts sixteen at a time.  Two sets of four
// warps serve NT tokens each; warp w of a set holds the chains of 16-byte pieces 8w .. 8w+7 of every 512-byte run (the
// chains 32w .. 32w+31), its lanes are 8 pieces x 4 expert groups, and a thread multiplies NT tokens by 4 experts for its
// four chains.  Every staged activation word feeds 4 chains of a thread and is broadcast to four groups; the router words
// come straight from L2 into registers, four steps ahead (600 cycles; one step ahead left the f32 pipe idle two thirds of
// the time; 4096 tokens x 256 experts x 3072: 271 us with one warp per expert pair, now 229).  fma.rn.f32x2 is two independent IEEE fmas, so the logits are bit-identical.
// The fold of a (token, expert) pair is the specified one: four chains per lane, then strides 16 and 8 across the warps
// (through shared memory) and 4, 2, 1 across the lanes.
constexpr int RT_THREADS = 256, RT_EXPERTS = 16; // experts of one pass
constexpr int RT_AHEAD = 4;

__device__ __forceinline__ void fma_f32x2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int NT>
__global__ void __launch_bounds__(RT_THREADS, 1)
route_logits_tiled_kernel(const float *__restrict__ router, const float *__restrict__ x, int t, int hidden, int n_expert,
                          int experts_per_block, float *__restrict__ logits) {
    extern __shared__ __align__(16) uint8_t rt_smem[];
    typedef ulonglong2 u2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = warp & 3, set = warp >> 2, piece = lane & 7, eg = lane >> 3;
    const int steps = hidden / 128, row = hidden / 4; // 16-byte words of a row
    const int t0 = blockIdx.x * 2 * NT, nt = min(2 * NT, t - t0);
    const int e_end = min(n_expert, (int)(blockIdx.y + 1) * experts_per_block);
    uint8_t *xs = rt_smem;
    float4 *fold = reinterpret_cast<float4 *>(rt_smem + (size_t)2 * NT * hidden * 4) + set * (4 * 4 * (NT / 4) * 32);
    {
        const uint8_t *src = reinterpret_cast<const uint8_t *>(x + (size_t)t0 * hidden);
        for (int i = threadIdx.x; i < nt * row; i += RT_THREADS) cp_async16(xs + (size_t)i * 16, src + (size_t)i * 16);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // this thread's piece of its four router rows, for this pass and the next (rows past the last one repeat it)
    const u2 *wr[4], *wx[4];
    auto rows = [&](const u2 *(&p)[4], int e0) {
#pragma unroll
        for (int e = 0; e < 4; e++)
            p[e] = reinterpret_cast<const u2 *>(router) + (size_t)min(e0 + 4 * eg + e, n_expert - 1) * row + 8 * w + piece;
    };
    int e0 = blockIdx.y * experts_per_block;
    rows(wr, e0);
    u2 wq[RT_AHEAD][4];
#pragma unroll
    for (int u = 0; u < RT_AHEAD; u++)
#pragma unroll
        for (int e = 0; e < 4; e++) wq[u][e] = u < steps ? __ldg(wr[e] + 32 * u) : make_ulonglong2(0ull, 0ull);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const u2 *xp = reinterpret_cast<const u2 *>(xs) + (size_t)set * NT * row + 8 * w + piece;
    for (; e0 < e_end; e0 += RT_EXPERTS) {
        rows(wx, e0 + RT_EXPERTS);
        unsigned long long acc[NT][4][2];
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][e][0] = acc[i][e][1] = 0ull;
        // steps is a multiple of RT_AHEAD (the launcher sees to it)
#pragma unroll 1
        for (int j = 0; j < steps; j += RT_AHEAD) {
#pragma unroll
            for (int u = 0; u < RT_AHEAD; u++) {
#pragma unroll
                for (int i = 0; i < NT; i++) {
                    const u2 xv = xp[(size_t)i * row + 32 * (j + u)];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        fma_f32x2(acc[i][e][0], xv.x, wq[u][e].x);
                        fma_f32x2(acc[i][e][1], xv.y, wq[u][e].y);
                    }
                }
                const bool more = j + RT_AHEAD < steps;
#pragma unroll
                for (int e = 0; e < 4; e++) wq[u][e] = __ldg((more ? wr[e] + 32 * (j + RT_AHEAD + u) : wx[e] + 32 * u));
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) wr[e] = wx[e];
        // fold: this lane's chains, then across the four warps of the set
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int h = 0; h < NT / 4; h++) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 a = *reinterpret_cast<const float2 *>(&acc[4 * h + i][e][0]), b = *reinterpret_cast<const float2 *>(&acc[4 * h + i][e][1]);
                    v[i] = __fadd_rn(__fadd_rn(a.x, a.y), __fadd_rn(b.x, b.y));
                }
                fold[((w * 4 + e) * (NT / 4) + h) * 32 + lane] = make_float4(v[0], v[1], v[2], v[3]);
            }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
        float r[NT]; // this warp finishes expert w of every group
#pragma unroll
        for (int h = 0; h < NT / 4; h++) {
            float4 p[4];
#pragma unroll
            for (int q = 0; q < 4; q++) p[q] = fold[((q * 4 + w) * (NT / 4) + h) * 32 + lane];
            r[4 * h + 0] = __fadd_rn(__fadd_rn(p[0].x, p[2].x), __fadd_rn(p[1].x, p[3].x));
            r[4 * h + 1] = __fadd_rn(__fadd_rn(p[0].y, p[2].y), __fadd_rn(p[1].y, p[3].y));
            r[4 * h + 2] = __fadd_rn(__fadd_rn(p[0].z, p[2].z), __fadd_rn(p[1].z, p[3].z));
            r[4 * h + 3] = __fadd_rn(__fadd_rn(p[0].w, p[2].w), __fadd_rn(p[1].w, p[3].w));
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory"); // the buffer is free for the next pass
        // strides 4, 2, 1: while there is more than one value, a step keeps half of them (by that bit of the lane)
        int n = NT;
#pragma unroll
        for (int st = 4; st >= 1; st >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool up = (lane & st) != 0;
#pragma unroll
                for (int i = 0; i < NT / 2; i++) {
                    if (i < n) {
                        const float keep = up ? r[i + n] : r[i], send = up ? r[i] : r[i + n];
                        r[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, st));
                    }
                }
            } else {
                r[0] = __fadd_rn(r[0], __shfl_xor_sync(0xffffffffu, r[0], st));
            }
        }
        // NT = 8: the lane's piece is the token; NT = 4: its upper two bits are, and the last step left both halves equal
        const int tok = set * NT + (NT == 8 ? piece : piece >> 1), ex = e0 + 4 * eg + w;
        if (tok < nt && ex < e_end && (NT == 8 || (piece & 1) == 0)) logits[(size_t)(t0 + tok) * n_expert + ex] = r[0];
    }
}

// One warp per token; scores staged in shared memory (2 * n_expert floats per warp).
__global__ void __launch_bounds__(ROUTE_WARPS * 32)
route_select_kernel(const float *__restrict__ logits, const float *__restrict__ bias, int t, int n_expert,
                    int top_k, float scale, int norm, uint32_t *__restrict__ ids, float *__restrict__ weights) {
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int token = blockIdx.x * ROUTE_WARPS + warp;
    if (token >= t) return;
    float *probs = smem + (size_t)warp * 2 * n_expert;
    float *sel = probs + n_expert;
    for (int e = lane; e < n_expert; e += 32) {
        const float p = lmoe_sigmoid_fixed(logits[(size_t)token * n_expert + e]);
        probs[e] = p;
        sel[e] = bias ? __fadd_rn(p, bias[e]) : p;
    }
    __syncwarp();
    lmoe_warp_select(sel, probs, n_expert, top_k, scale, norm, ids + (size_t)token * top_k,
                     weights + (size_t)token * top_k, lane);
}

} // namespace

cudaError_t launch_route_logits(const float *router, const float *x, int t, int hidden, int n_expert,
                                float *logits, cudaStream_t s) {
    if (t == 0) return cudaSuccess;
    const unsigned gx = (unsigned)((n_expert + ROUTE_WARPS - 1) / ROUTE_WARPS);
    // 16 tokens per block where their rows fit beside the fold buffer (hidden <= 3072), else 8
    const int nt = 16 * hidden * 4 + 2 * 16384 <= 227 * 1024 ? 8 : 4;
    const int smem = 2 * nt * hidden * 4 + 2 * (nt / 4) * 8192;
    if (t > 64 && hidden % (128 * RT_AHEAD) == 0 && smem <= 227 * 1024) {
        static int sms_of[64] = {0}; // per device: SM count, and the shared-memory opt-in done once
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
        if (!sms_of[dev]) {
            int n = 0;
            if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
            cudaFuncSetAttribute(route_logits_tiled_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            cudaFuncSetAttribute(route_logits_tiled_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            sms_of[dev] = n;
        }
        // (Up to 64 tokens a warp per expert row covers the device better: 7 us against 9 at 16 tokens.)
        // One block per SM at a time.  The experts are split over blocks until the device is covered, and further where that
        // fills the last wave better; a block repeats the staging of its tokens (about a tenth of a full pass over 256
        // experts), hence the weight of one and a half passes below.
        const int tiles = (t + 2 * nt - 1) / (2 * nt), passes = (n_expert + RT_EXPERTS - 1) / RT_EXPERTS;
        int best_ppb = passes;
        double best = 1e30;
        for (int ppb = passes; ppb >= 1; ppb--) {
            const int64_t blocks = (int64_t)tiles * ((passes + ppb - 1) / ppb);
            const double cost = (double)((blocks + sms_of[dev] - 1) / sms_of[dev]) * (ppb + 1.5);
            if (cost < best) { best = cost; best_ppb = ppb; }
        }
        const dim3 grid((unsigned)tiles, (unsigned)((passes + best_ppb - 1) / best_ppb));
        if (nt == 8)
            route_logits_tiled_kernel<8><<<grid, RT_THREADS, smem, s>>>(router, x, t, hidden, n_expert, best_ppb * RT_EXPERTS, logits);
        else
            route_logits_tiled_kernel<4><<<grid, RT_THREADS, smem, s>>>(router, x, t, hidden, n_expert, best_ppb * RT_EXPERTS, logits);
    } else if (t <= 2) {
        route_logits_kernel<1><<<dim3(gx, t), ROUTE_WARPS * 32, 0, s>>>(router, x, t, hidden, n_expert, logits);
    } else {
        route_logits_kernel<4><<<dim3(gx, (t + 3) / 4), ROUTE_WARPS * 32, 0, s>>>(router, x, t, hidden, n_expert, logits);
    }
    return cudaGetLastError();
}

cudaError_t launch_route_select(const float *logits, const float *bias, int t, int n_expert, int top_k,
                                float scale, int norm, uint32_t *ids, float *weights, cudaStream_t s) {
    if (t == 0) return cudaSuccess;
    const size_t smem = (size_t)ROUTE_WARPS * 2 * n_expert * sizeof(float);
    const unsigned grid = (unsigned)((t + ROUTE_WARPS - 1) / ROUTE_WARPS);
    route_select_kernel<<<grid, ROUTE_WARPS * 32, smem, s>>>(logits, bias, t, n_expert, top_k, scale, norm, ids,
                                                             weights);
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
