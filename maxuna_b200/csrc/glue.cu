// Small kernels around the expert matmuls: silu(g)*u, the weighted top-k
// combine, and the per-expert token-slot map ("map0").
// Reference: src/ops/silu_mul.metal:57-72, src/ops/combine.metal:70-133,
// src/ops/mm_id.metal:207-269.
#include "common.cuh"
#include "route_math.cuh"

namespace {

__device__ __forceinline__ float silu_mul(float a, float u) {
    return __fmul_rn(__fdiv_rn(a, __fadd_rn(1.0f, expf(-a))), u); // two separate roundings, then the product
}
// Four values a thread: as 16-byte words where the pointers allow it (VEC; the last thread takes what is left of them one by
// one), else 256 apart.  One value a thread (PER = 1) is the shorter start of a small unaligned call (4096 values 1.4 us, four a
// thread 2.2) and half as fast on a large one.  5120 x 1024 values 6.7 us, unaligned 9.2, one a thread 22.
template <bool VEC, int PER>
__global__ void silu_mul_kernel(const float *__restrict__ g, const float *__restrict__ u, int64_t n,
                                float *__restrict__ out) {
    pdl_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (VEC && 4 * i + 4 <= n) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(g) + i), b = __ldg(reinterpret_cast<const float4 *>(u) + i);
        reinterpret_cast<float4 *>(out)[i] = make_float4(silu_mul(a.x, b.x), silu_mul(a.y, b.y), silu_mul(a.z, b.z), silu_mul(a.w, b.w));
    } else if (VEC) {
        for (int64_t j = 4 * i; j < n; j++) out[j] = silu_mul(g[j], u[j]);
    } else {
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int64_t j = ((int64_t)blockIdx.x * PER + q) * blockDim.x + threadIdx.x;
            if (j < n) out[j] = silu_mul(g[j], u[j]);
        }
    }
}

// Range guard of a row before it is rounded to f16: its L2 norm (clamped), and the row times 2^15 over the norm.  One warp a
// row; the second read comes from L1.  5120 x 1024 values: 15 us,
// as six element-wise steps 47.
__global__ void __launch_bounds__(256) l2_rescale_kernel(const float *__restrict__ a, int64_t rows, int n, float *__restrict__ out,
                                                         float *__restrict__ l2) {
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float *ar = a + row * n;
    float *orow = out + row * n;
    float ss = 0.f;
#pragma unroll 4
    for (int i = lane; i < n; i += 32) ss = __fmaf_rn(ar[i], ar[i], ss);
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float norm = isnan(ss) ? ss : fminf(fmaxf(sqrtf(ss), 1e-8f), 1e30f);
#pragma unroll 4
    for (int i = lane; i < n; i += 32) orow[i] = __fdiv_rn(__fmul_rn(ar[i], 32768.0f), norm);
    if (lane == 0) l2[row] = norm;
}

// Eight values of a row -> their place in the tile order, divided by the row's norm and rounded to f16 as gather_tiles_kernel does.
__device__ __forceinline__ void rescale_chunk(const float *a, int ci, float norm, int p, int n, int nt, uint8_t *__restrict__ act) {
    const float4 b = *reinterpret_cast<const float4 *>(a + ci * 8), c = *reinterpret_cast<const float4 *>(a + ci * 8 + 4);
    const float v[8] = {b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
    float q[8];
#pragma unroll
    for (int j = 0; j < 8; j++) q[j] = __fdiv_rn(__fmul_rn(v[j], 32768.0f), norm);
    __align__(16) __half2 h[4] = {__floats2half2_rn(q[0], q[2]), __floats2half2_rn(q[1], q[3]), __floats2half2_rn(q[4], q[6]),
                                  __floats2half2_rn(q[5], q[7])};
    const size_t off = (((size_t)(p / nt) * (n / 64) + (ci >> 3)) * nt + (p % nt)) * 128 + ((size_t)((ci & 7) ^ (p & 7)) << 4);
    *reinterpret_cast<uint4 *>(act + off) = *reinterpret_cast<const uint4 *>(h);
}
__device__ __forceinline__ float row_norm(float ss) { // of a lane's share of the squares
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    return isnan(ss) ? ss : fminf(fmaxf(sqrtf(ss), 1e-8f), 1e30f);
}

// Both steps at once, a block a row: the bits of silu_mul_kernel and l2_rescale_kernel.  The activations stay in shared memory
// between the two passes instead of going through memory three times (5120 x 1024 values, with a cold cache: 12 + 16 + 11 us in
// three kernels, 25 here).  Bound by memory from rows of 4096 on; below, by the chain load, sum, divide of a block.  The squares are
// summed by one warp, in l2_rescale_kernel's order.  (A warp a row left the wide rows few loads in flight, as a warp's row stays
// in shared memory: 5120 rows of 256 / 1024 / 4096 / 12288 values 14 / 33 / 237 / 2006 us, a block a row 12 / 25 / 61 / 177.)
__global__ void __launch_bounds__(256) silu_rescale_tiles_kernel(const float *__restrict__ g, const float *__restrict__ u,
                                                                 const int32_t *__restrict__ pos, int n, int nt, uint8_t *__restrict__ act,
                                                                 float *__restrict__ l2, float *__restrict__ y, int n_y) {
    pdl_begin();
    extern __shared__ __align__(16) float sr_row[];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int64_t row = blockIdx.x;
    const int p = pos[row];
    if (p < 0) {
        for (int i = tid; i < n_y; i += nthr) y[row * n_y + i] = 0.f;
        if (tid == 0) l2[row] = 1.0f;
        return;
    }
    const float4 *gr = reinterpret_cast<const float4 *>(g + row * n), *ur = reinterpret_cast<const float4 *>(u + row * n);
#pragma unroll 2
    for (int i = tid; i < n / 4; i += nthr) {
        const float4 b = __ldg(gr + i), c = __ldg(ur + i);
        reinterpret_cast<float4 *>(sr_row)[i] = make_float4(silu_mul(b.x, c.x), silu_mul(b.y, c.y), silu_mul(b.z, c.z), silu_mul(b.w, c.w));
    }
    __syncthreads();
    if (tid < 32) {
        float ss = 0.f;
#pragma unroll 8
        for (int i = tid; i < n; i += 32) ss = __fmaf_rn(sr_row[i], sr_row[i], ss);
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (tid == 0) l2[row] = isnan(ss) ? ss : fminf(fmaxf(sqrtf(ss), 1e-8f), 1e30f);
    }
    __syncthreads();
    const float norm = l2[row]; // (shared memory may be the row's to the last byte)
    for (int ci = tid; ci < n / 8; ci += nthr) {
        const float4 b = *reinterpret_cast<const float4 *>(sr_row + ci * 8), c = *reinterpret_cast<const float4 *>(sr_row + ci * 8 + 4);
        const float v[8] = {b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
        float q[8];
#pragma unroll
        for (int j = 0; j < 8; j++) q[j] = __fdiv_rn(__fmul_rn(v[j], 32768.0f), norm);
        // rounded to f16 as gather_tiles_kernel does
        __align__(16) __half2 h[4] = {__floats2half2_rn(q[0], q[2]), __floats2half2_rn(q[1], q[3]), __floats2half2_rn(q[4], q[6]),
                                      __floats2half2_rn(q[5], q[7])};
        const size_t off = (((size_t)(p / nt) * (n / 64) + (ci >> 3)) * nt + (p % nt)) * 128 + ((size_t)((ci & 7) ^ (p & 7)) << 4);
        *reinterpret_cast<uint4 *>(act + off) = *reinterpret_cast<const uint4 *>(h);
    }
}

__global__ void add_inplace_kernel(float *__restrict__ out, const float *__restrict__ b, int64_t n) {
    pdl_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __fadd_rn(out[i], b[i]);
}

// V consecutive columns of one row per thread (four where rows are whole 16-byte words). The top_k terms are summed in the
// order of the reference's launch geometry: k strided over W lanes, then a butterfly. 512 rows of 10 x 3072: 43 -> 20 us.
// CHECKED: `flag` is the device flag of the products summed here; once it is set the rows are NaN, never a wrong finite sum.
template <int W, int V, bool CHECKED>
__global__ void combine_kernel(const float *__restrict__ down, const float *__restrict__ col_l2,
                               const float *__restrict__ w, int seq, int top_k, int n_out,
                               float *__restrict__ out, const uint32_t *flag) {
    pdl_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int nv = n_out / V;
    if (i >= (int64_t)seq * nv) return;
    if (CHECKED && *flag != 0u) {
#pragma unroll
        for (int q = 0; q < V; q++) out[i * V + q] = __int_as_float(0x7fc00000);
        return;
    }
    const int s = (int)(i / nv), c = (int)(i % nv) * V;
    const float *dp = down + (size_t)s * top_k * n_out + c, *wp = w + (size_t)s * top_k;
    alignas(16) float v[W][V];
#pragma unroll
    for (int l = 0; l < W; l++)
#pragma unroll
        for (int q = 0; q < V; q++) v[l][q] = 0.0f;
    for (int k0 = 0; k0 < top_k; k0 += W) {
#pragma unroll
        for (int l = 0; l < W; l++) {
            const int k = k0 + l;
            if (k >= top_k) break;
            alignas(16) float d[V];
            if (V == 4) *reinterpret_cast<float4 *>(d) = __ldg(reinterpret_cast<const float4 *>(dp + (size_t)k * n_out));
            else d[0] = __ldg(dp + (size_t)k * n_out);
#pragma unroll
            for (int q = 0; q < V; q++) {
                if (col_l2) {
                    d[q] = __fmul_rn(d[q], col_l2[(size_t)s * top_k + k]);
                    d[q] = __fmul_rn(d[q], 0x1p-15f);
                }
                v[l][q] = __fadd_rn(v[l][q], __fmul_rn(d[q], wp[k]));
            }
        }
    }
#pragma unroll
    for (int off = W / 2; off >= 1; off >>= 1)
#pragma unroll
        for (int l = 0; l < off; l++)
#pragma unroll
            for (int q = 0; q < V; q++) v[l][q] = __fadd_rn(v[l][q], v[l + off][q]);
    if (V == 4) reinterpret_cast<float4 *>(out)[i] = *reinterpret_cast<const float4 *>(v[0]);
    else out[i] = v[0][0];
}

// One block of NT threads per expert: scan the tokens in chunks of 4 NT (four consecutive tokens per thread), keep the
// token order, write flat ids `token*top_k + slot`.  VEC: the four tokens' ids as top_k 16-byte words (t a multiple of
// four, `ids` aligned): a quarter of the load instructions, which are what the scan spends its time on.
template <bool VEC, int NT>
__global__ void __launch_bounds__(NT)
map0_kernel(const uint32_t *__restrict__ ids, int t, int top_k, int n_expert, uint32_t *__restrict__ tpe,
            int32_t *__restrict__ ids_map) {
    pdl_begin();
    __shared__ int warp_count[NT / 32];
    __shared__ int base;
    const int e = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    int32_t *dst = ids_map + (size_t)e * t;
    for (int t0 = 0; t0 < t; t0 += 4 * NT) {
        int slot[4] = {-1, -1, -1, -1}, mine = 0;
        const int tok0 = t0 + 4 * (int)threadIdx.x;
        if (VEC) {
            if (tok0 < t) {
                const uint4 *p = reinterpret_cast<const uint4 *>(ids + (size_t)tok0 * top_k);
                int j = 0, s = 0; // token and slot of the next id
                for (int i = 0; i < top_k; i++) {
                    const uint4 v = __ldg(p + i);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (w[q] == (uint32_t)e) {
#pragma unroll
                            for (int jj = 0; jj < 4; jj++)
                                if (jj == j && slot[jj] < 0) slot[jj] = s;
                        }
                        if (++s == top_k) { s = 0; j++; }
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int token = tok0 + j;
                if (token < t) {
                    for (int s = 0; s < top_k; s++)
                        if (ids[(size_t)token * top_k + s] == (uint32_t)e) { slot[j] = s; break; }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) mine += slot[j] >= 0;
        // exclusive prefix of the per-thread counts inside the warp, then over the warps
        int pre = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        if (lane == 31) warp_count[warp] = pre;
        __syncthreads();
        int off = base + pre - mine;
        for (int wv = 0; wv < warp; wv++) off += warp_count[wv];
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (slot[j] >= 0) dst[off++] = (t0 + 4 * (int)threadIdx.x + j) * top_k + slot[j];
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int wv = 0; wv < NT / 32; wv++) tot += warp_count[wv];
            base += tot;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) tpe[e] = (uint32_t)base;
}

// RMS norm of one row per warp (`ffn_norm`, src/model.rs:340): out = (x * inv) * weight with
// inv = 1 / sqrt(sum(x^2) / hidden + eps).  The sum of squares runs in the router's reduction order
// (128 fmaf chains over elements c, c + 128, ..., folded per lane and by the warp butterfly), so the
// router input - and with it the expert selection - does not depend on the launch geometry.
__global__ void __launch_bounds__(256) rms_norm_kernel(const float *__restrict__ x, const float *__restrict__ w, float eps,
                                                       int t, int hidden, float *__restrict__ out) {
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= t) return;
    const float *xr = x + (size_t)row * hidden;
    float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
    for (int i = lane * 4; i < hidden; i += 128) {
        const float4 v = *reinterpret_cast<const float4 *>(xr + i);
        p0 = __fmaf_rn(v.x, v.x, p0);
        p1 = __fmaf_rn(v.y, v.y, p1);
        p2 = __fmaf_rn(v.z, v.z, p2);
        p3 = __fmaf_rn(v.w, v.w, p3);
    }
    const float ss = lmoe_router_fold(p0, p1, p2, p3);
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)hidden), eps)));
    float *orow = out + (size_t)row * hidden;
    for (int i = lane * 4; i < hidden; i += 128) {
        const float4 v = *reinterpret_cast<const float4 *>(xr + i);
        const float4 g = __ldg(reinterpret_cast<const float4 *>(w + i));
        float4 o;
        o.x = __fmul_rn(__fmul_rn(v.x, inv), g.x);
        o.y = __fmul_rn(__fmul_rn(v.y, inv), g.y);
        o.z = __fmul_rn(__fmul_rn(v.z, inv), g.z);
        o.w = __fmul_rn(__fmul_rn(v.w, inv), g.w);
        *reinterpret_cast<float4 *>(orow + i) = o;
    }
}

} // namespace

cudaError_t launch_rms_norm(const float *x, const float *w, float eps, int64_t t, int hidden, float *out, cudaStream_t s) {
    if (t == 0) return cudaSuccess;
    launch_pdl(rms_norm_kernel, (unsigned)((t + 7) / 8), 256, 0, s, x, w, eps, (int)t, hidden, out);
    return cudaGetLastError();
}

static bool aligned16_all(const void *a, const void *b, const void *c) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) == 0;
}

cudaError_t launch_silu_mul(const float *g, const float *u, int64_t n, float *out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const unsigned g4 = (unsigned)(((n + 3) / 4 + 255) / 256);
    if (aligned16_all(g, u, out)) launch_pdl(silu_mul_kernel<true, 4>, g4, 256, 0, s, g, u, n, out);
    else if (n >= 1 << 18) launch_pdl(silu_mul_kernel<false, 4>, g4, 256, 0, s, g, u, n, out);
    else launch_pdl(silu_mul_kernel<false, 1>, (unsigned)((n + 255) / 256), 256, 0, s, g, u, n, out);
    return cudaGetLastError();
}

cudaError_t launch_silu_rescale_tiles(const float *g, const float *u, const int32_t *pos, int64_t rows, int n, int nt, void *act, float *l2,
                                      float *y, int n_y, cudaStream_t s) {
    if (rows == 0) return cudaSuccess;
    if (n > LMOE_FFN_MM_MAX_FF) return cudaErrorInvalidValue; // a row in the shared memory that needs no opt-in
    launch_pdl(silu_rescale_tiles_kernel, (unsigned)rows, n < 1024 ? n / 4 : 256, (size_t)n * 4, s, g, u, pos, n, nt, static_cast<uint8_t *>(act),
               l2, y, n_y);
    return cudaGetLastError();
}

cudaError_t launch_l2_rescale(const float *a, int64_t rows, int n, float *out, float *l2, cudaStream_t s) {
    if (rows == 0) return cudaSuccess;
    launch_pdl(l2_rescale_kernel, (unsigned)((rows + 7) / 8), 256, 0, s, a, rows, n, out, l2);
    return cudaGetLastError();
}

cudaError_t launch_add_inplace(float *out, const float *b, int64_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_pdl(add_inplace_kernel, (unsigned)((n + 255) / 256), 256, 0, s, out, b, n);
    return cudaGetLastError();
}

template <int W, bool CHECKED>
static void combine_launch(const float *down, const float *col_l2, const float *w, int seq, int top_k, int n_out, float *out, cudaStream_t s,
                           const uint32_t *flag) {
    const int64_t n = (int64_t)seq * n_out;
    if (n_out % 4 == 0 && aligned16_all(down, out, nullptr))
        launch_pdl(combine_kernel<W, 4, CHECKED>, (unsigned)((n / 4 + 127) / 128), 128, 0, s, down, col_l2, w, seq, top_k, n_out, out, flag);
    else
        launch_pdl(combine_kernel<W, 1, CHECKED>, (unsigned)((n + 255) / 256), 256, 0, s, down, col_l2, w, seq, top_k, n_out, out, flag);
}

cudaError_t launch_combine(const float *down, const float *col_l2, const float *w, int seq, int top_k,
                           int n_out, float *out, cudaStream_t s, const uint32_t *flag) {
    if ((int64_t)seq * n_out == 0) return cudaSuccess;
    int width = 1;
    while (width < top_k / 2) width <<= 1;
#define COMBINE(W) (flag ? combine_launch<W, true> : combine_launch<W, false>)(down, col_l2, w, seq, top_k, n_out, out, s, flag)
    switch (width) {
    case 1: COMBINE(1); break;
    case 2: COMBINE(2); break;
    case 4: COMBINE(4); break;
    case 8: COMBINE(8); break;
    case 16: COMBINE(16); break;
    default: COMBINE(32); break;
    }
#undef COMBINE
    return cudaGetLastError();
}

cudaError_t launch_map0(const uint32_t *ids, int t, int top_k, int n_expert, uint32_t *tpe, int32_t *ids_map,
                        cudaStream_t s) {
    if (n_expert == 0) return cudaSuccess;
    // A chunk is a chain of latencies, and the blocks of 256 experts are resident at once in either size: as many threads as one
    // or a few chunks need (256 experts, top-10, 2048 / 4096 / 16384 tokens: 7.8 / 14.5 / 53 us with
    // 256 threads, 6.0 / 8.6 / 33 with 1024).
    const bool vec = t % 4 == 0 && (reinterpret_cast<uintptr_t>(ids) & 15u) == 0;
    if (t <= 1024) launch_pdl(vec ? map0_kernel<true, 256> : map0_kernel<false, 256>, n_expert, 256, 0, s, ids, t, top_k, n_expert, tpe, ids_map);
    else launch_pdl(vec ? map0_kernel<true, 1024> : map0_kernel<false, 1024>, n_expert, 1024, 0, s, ids, t, top_k, n_expert, tpe, ids_map);
    return cudaGetLastError();
}

// Expert ids of the whole block -> ids relative to the experts [first, first + count) resident on one rank;
// every other id (other ranks' experts, or already-empty slots) becomes the empty-slot id `count`.
__global__ void ep_localize_ids_kernel(const uint32_t *__restrict__ ids, int64_t n, uint32_t first, uint32_t count,
                                       uint32_t *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t e = ids[i] - first; // wraps for ids below `first`
    out[i] = e < count ? e : count;
}

cudaError_t launch_ep_localize_ids(const uint32_t *ids, int64_t n, uint32_t first, uint32_t count, uint32_t *out,
                                   cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    ep_localize_ids_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ids, n, first, count, out);
    return cudaGetLastError();
}
