// Prefill path: routing, per-expert row lists, grouped tensor-core GEMMs for
// gate / up / down, SwiGLU with the f16 range guard, fixed-order combine, shared expert.
// Reference: the mm_id branch of `FusedExperts::forward`, src/moe.rs:236-323, and
// `MoeBlock::forward`, src/moe.rs:73-78.
#include "fused.cuh"

// mm_id.cu
bool mm_id_kernel_available(int dtype, int64_t n_out, int64_t k);
MmRows mm_rows(int64_t rows, int64_t extra, int64_t n_expert);
size_t mm_tiles_bytes(const MmRows &R);
size_t mm_tiled_bytes(const MmRows &R, int64_t k);
lmoe_status launch_gather_tiles(const MmRows &R, const void *x, int x_f16, int x_per_row, int top_k, int k, const uint32_t *tpe,
                                const int32_t *ids_map, int64_t map_stride, void *tiles_ws, void *xt, int32_t *pos, int32_t *spos,
                                int32_t *sfid, cudaStream_t s);
size_t mm_src_bytes(const MmRows &R);
lmoe_status launch_stage_rows(const MmRows &R, const void *x, int x_f16, int64_t x_rows, int top_k, int k, const uint32_t *tpe,
                              const int32_t *ids_map, int64_t map_stride, void *tiles_ws, void *xh, int32_t *src, int32_t *pos,
                              int32_t *spos, int32_t *sfid, cudaStream_t s);
lmoe_status launch_mm_gateup(const MmRows &R, const lmoe_expert_stack *gate, const lmoe_expert_stack *up, const lmoe_expert_stack *sh_gate,
                             const lmoe_expert_stack *sh_up, const void *xh, const int32_t *src, const int32_t *ids_map, int64_t map_stride, float *act,
                             int sorted, void *tiles_ws, uint32_t *flag, cudaStream_t stream);
lmoe_status launch_mm_id(const MmRows &R, const lmoe_expert_stack *st, const lmoe_expert_stack *shared, const void *xt,
                         const int32_t *ids_map, int64_t map_stride, const float *row_scale, float *out, int sorted, void *tiles_ws,
                         uint32_t *flag, cudaStream_t stream);

namespace {

// One warp per row: act = silu(g) * u; l2 = clamp(||act||, 1e-8, 1e30); the f16 operand of the
// down projection is act * 32768 / l2 (src/moe.rs:292-302), written in the grouped GEMM's tile
// order (row tile pos / nt, row pos % nt, 128-byte swizzle, groups of 8 as [0 2 1 3 4 6 5 7]);
// scale[row] = l2 * 2^-15 * weight[row] undoes it in the down epilogue together with the
// routing weight (src/ops/combine.metal:102-133).
// A row that no list names (pos < 0) is a zero row of `y`.
__device__ __forceinline__ void zero_row(float *y, int hidden, int lane) {
    for (int i = lane; i < hidden; i += 32) y[i] = 0.f;
}
__global__ void __launch_bounds__(256) swiglu_rows_kernel(const float *__restrict__ g, const float *__restrict__ u,
                                                          const float *__restrict__ w, const int32_t *__restrict__ pos,
                                                          int64_t rows, int ff, int nt, uint8_t *__restrict__ act,
                                                          float *__restrict__ scale, float *__restrict__ y, int hidden) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int p = pos[row];
    if (p < 0) { zero_row(y + row * hidden, hidden, lane); return; }
    const float *gr = g + row * ff, *ur = u + row * ff;
    float ss = 0.f;
    for (int i = lane * 8; i < ff; i += 256) {
        const float4 g0 = *reinterpret_cast<const float4 *>(gr + i), g1 = *reinterpret_cast<const float4 *>(gr + i + 4);
        const float4 u0 = *reinterpret_cast<const float4 *>(ur + i), u1 = *reinterpret_cast<const float4 *>(ur + i + 4);
        const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        const float uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float a = __fmul_rn(__fdiv_rn(gv[j], __fadd_rn(1.0f, expf(-gv[j]))), uv[j]);
            ss += a * a;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float l2 = fminf(fmaxf(sqrtf(ss), 1e-8f), 1e30f);
    const float k = 32768.0f / l2;
    for (int i = lane * 8; i < ff; i += 256) {
        const float4 g0 = *reinterpret_cast<const float4 *>(gr + i), g1 = *reinterpret_cast<const float4 *>(gr + i + 4);
        const float4 u0 = *reinterpret_cast<const float4 *>(ur + i), u1 = *reinterpret_cast<const float4 *>(ur + i + 4);
        const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        const float uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
        float a[8];
#pragma unroll
        for (int j = 0; j < 8; j++) a[j] = __fmul_rn(__fdiv_rn(gv[j], __fadd_rn(1.0f, expf(-gv[j]))), uv[j]) * k;
        __align__(16) __half2 h[4] = {__floats2half2_rn(a[0], a[2]), __floats2half2_rn(a[1], a[3]),
                                      __floats2half2_rn(a[4], a[6]), __floats2half2_rn(a[5], a[7])};
        const int ci = i >> 3;
        const size_t off = (((size_t)(p / nt) * (ff / 64) + (ci >> 3)) * nt + (p % nt)) * 128 +
                           ((size_t)((ci & 7) ^ (p & 7)) << 4);
        *reinterpret_cast<uint4 *>(act + off) = *reinterpret_cast<const uint4 *>(h);
    }
    if (lane == 0) scale[row] = l2 * 0x1p-15f * (w ? w[row] : 1.0f);
}

// Same range guard for an activation that is already silu(g)*u (f32): l2, rescale, f16, tile order.
// With `sfid` the rows of `a` (and of `scale`) are in expert-sorted order and sfid[row] is the flat id; ids from `routed` on
// are the shared expert's rows, which carry no routing weight.
__global__ void __launch_bounds__(256) rescale_rows_kernel(const float *__restrict__ a, const float *__restrict__ w,
                                                           const int32_t *__restrict__ pos, const int32_t *__restrict__ sfid,
                                                           int64_t rows, int64_t routed, int ff, int nt, uint8_t *__restrict__ act,
                                                           float *__restrict__ scale, float *__restrict__ y, int hidden) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int64_t fid = sfid ? sfid[row] : row;
    if (fid < 0) return;                                   // no routed row here (masked slots leave a tail unused)
    const int p = pos[fid];
    if (p < 0) { zero_row(y + row * hidden, hidden, lane); return; } // (rows by flat id only)
    const float *ar = a + row * ff;
    float ss = 0.f;
    for (int i = lane * 8; i < ff; i += 256) {
        const float4 a0 = *reinterpret_cast<const float4 *>(ar + i), a1 = *reinterpret_cast<const float4 *>(ar + i + 4);
        ss += a0.x * a0.x + a0.y * a0.y + a0.z * a0.z + a0.w * a0.w + a1.x * a1.x + a1.y * a1.y + a1.z * a1.z + a1.w * a1.w;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float l2 = fminf(fmaxf(sqrtf(ss), 1e-8f), 1e30f);
    const float k = 32768.0f / l2;
    for (int i = lane * 8; i < ff; i += 256) {
        const float4 a0 = *reinterpret_cast<const float4 *>(ar + i), a1 = *reinterpret_cast<const float4 *>(ar + i + 4);
        __align__(16) __half2 h[4] = {__floats2half2_rn(a0.x * k, a0.z * k), __floats2half2_rn(a0.y * k, a0.w * k),
                                      __floats2half2_rn(a1.x * k, a1.z * k), __floats2half2_rn(a1.y * k, a1.w * k)};
        const int ci = i >> 3;
        const size_t off = (((size_t)(p / nt) * (ff / 64) + (ci >> 3)) * nt + (p % nt)) * 128 +
                           ((size_t)((ci & 7) ^ (p & 7)) << 4);
        *reinterpret_cast<uint4 *>(act + off) = *reinterpret_cast<const uint4 *>(h);
    }
    if (lane == 0) scale[row] = l2 * 0x1p-15f * (w && fid < routed ? w[fid] : 1.0f);
}

// out[t, c] = sum over slots (in slot order) of y[t, s, c], then + shared[t, c], then + residual[t, c].
__global__ void sum_slots_kernel(const float *__restrict__ y, const float *__restrict__ shared,
                                 const float *__restrict__ residual, int64_t t, int top_k, int n4, float *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= t * n4) return;
    const int64_t tok = i / n4, c = i - tok * n4;
    const float4 *yp = reinterpret_cast<const float4 *>(y) + tok * top_k * n4 + c;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < top_k; k++) {
        const float4 v = yp[(int64_t)k * n4];
        s.x = __fadd_rn(s.x, v.x); s.y = __fadd_rn(s.y, v.y); s.z = __fadd_rn(s.z, v.z); s.w = __fadd_rn(s.w, v.w);
    }
    if (shared) {
        const float4 v = reinterpret_cast<const float4 *>(shared)[i];
        s.x = __fadd_rn(s.x, v.x); s.y = __fadd_rn(s.y, v.y); s.z = __fadd_rn(s.z, v.z); s.w = __fadd_rn(s.w, v.w);
    }
    if (residual) {
        const float4 v = reinterpret_cast<const float4 *>(residual)[i];
        s.x = __fadd_rn(s.x, v.x); s.y = __fadd_rn(s.y, v.y); s.z = __fadd_rn(s.z, v.z); s.w = __fadd_rn(s.w, v.w);
    }
    reinterpret_cast<float4 *>(out)[i] = s;
}

// Same sum when the partial rows are unscaled and in expert-sorted order: row spos[flat id] of `y`
// times scale[that row]; likewise for the shared expert's rows, then + residual.  A negative position marks an empty slot.
struct SumRows {
    const float *y, *scale;
    const int32_t *spos;
    const float *shared, *sh_scale;
    const int32_t *sh_spos;
    const float *residual;
    int64_t t;
    int top_k, n4;
    float *out;
    __device__ __forceinline__ void put(int64_t i, float4 s) const {
        if (residual) {
            const float4 v = reinterpret_cast<const float4 *>(residual)[i];
            s.x = __fadd_rn(s.x, v.x); s.y = __fadd_rn(s.y, v.y); s.z = __fadd_rn(s.z, v.z); s.w = __fadd_rn(s.w, v.w);
        }
        reinterpret_cast<float4 *>(out)[i] = s;
    }
    __device__ __forceinline__ static void add(float4 &s, const float4 v, float sc) {
        s.x = __fadd_rn(s.x, __fmul_rn(v.x, sc)); s.y = __fadd_rn(s.y, __fmul_rn(v.y, sc));
        s.z = __fadd_rn(s.z, __fmul_rn(v.z, sc)); s.w = __fadd_rn(s.w, __fmul_rn(v.w, sc));
    }
    // four columns of a token; twelve rows' loads are in flight
    __device__ __forceinline__ void columns(int64_t tok, int64_t c) const {
        const int32_t *sp = spos + tok * top_k;
        const int n = top_k + (shared ? 1 : 0);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = 0; k0 < n; k0 += 12) {
            float4 v[12];
            float sc[12];
            uint32_t present = 0u;
#pragma unroll
            for (int j = 0; j < 12; j++) {
                const int k = k0 + j;
                const bool sh = k == top_k;
                const int64_t r = k >= n ? -1 : (sh ? (sh_spos ? sh_spos[tok] : tok) : sp[k]);
                const float *base = sh ? shared : y, *sb = sh ? sh_scale : scale;
                sc[j] = r >= 0 && sb ? sb[r] : 1.0f;
                v[j] = r >= 0 ? __ldcs(reinterpret_cast<const float4 *>(base) + r * n4 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                present |= (uint32_t)(r >= 0) << j;
            }
#pragma unroll
            for (int j = 0; j < 12; j++)
                if (present & (1u << j)) add(s, v[j], sc[j]);
        }
        put(tok * n4 + c, s);
    }
};
__global__ void __launch_bounds__(256) sum_sorted_kernel(const SumRows R) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R.t * R.n4) return;
    const int64_t tok = i / R.n4;
    R.columns(tok, i - tok * R.n4);
}
// A block a token: up to twelve rows' places and scales, which the loads wait for, are read once for all of its columns.
__global__ void __launch_bounds__(256, 3) sum_tokens_kernel(const SumRows R) {
    const int64_t tok = blockIdx.x;
    const int n = R.top_k + (R.shared ? 1 : 0);
    if (n > 12) {
        for (int c = threadIdx.x; c < R.n4; c += 256) R.columns(tok, c);
        return;
    }
    int row[12];
    float sc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const bool sh = k == R.top_k;
        row[k] = k >= n ? -1 : (sh ? (R.sh_spos ? R.sh_spos[tok] : (int)tok) : R.spos[tok * R.top_k + k]);
        const float *sb = sh ? R.sh_scale : R.scale;
        sc[k] = row[k] >= 0 && sb ? sb[row[k]] : 1.0f;
    }
    for (int c = threadIdx.x; c < R.n4; c += 256) {
        float4 v[12];
#pragma unroll
        for (int k = 0; k < 12; k++)
            v[k] = row[k] >= 0 ? __ldcs(reinterpret_cast<const float4 *>(k == R.top_k ? R.shared : R.y) + (int64_t)row[k] * R.n4 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 12; k++)
            if (row[k] >= 0) SumRows::add(s, v[k], sc[k]);
        R.put(tok * R.n4 + c, s);
    }
}
// Which of the two, us for (columns over the whole grid) / (a block a token), cold L2, 11 rows a token:
//   hidden              512          1024         1536         2048         3072         7168
//   1024 tokens    14.3 / 14.3  18.4 / 16.4  22.5 / 22.5  26.6 / 26.6  34.8 / 34.8  69.6 / 67.6
//   2048 tokens    18.5 / 20.5  26.6 / 24.6  34.8 / 34.8  45.1 / 41.0  61.4 / 57.3   129 / 119
//   16384 tokens   77.8 / 94.1   150 / 137    217 / 200    289 / 252    428 / 373
// Rows of fewer than 2048 columns leave threads without work, or gain with some numbers of rows and lose with others (16384 tokens of 1536, 2 / 5 / 9 / 11 rows
// 131 / 135, 145 / 152, 178 / 180, 217 / 200; of 1280 111 / 129, 123 / 145, 150 / 168, 182 / 182).  More than twelve rows gain from 2048 tokens on (17 rows of 3072, 1024 /
// 2048 / 4096 tokens 51.2 / 51.2, 92.2 / 85.9, 172 / 162; 24 rows of 7168, 1024 tokens 131 / 135).
bool sum_by_token(int64_t t, int64_t n4, int n) { return t >= (n > 12 ? 2048 : 1024) && n4 >= 512 && t * n4 >= 768 * 1024; }
cudaError_t launch_sum_sorted(const SumRows &R, cudaStream_t s) {
    if (sum_by_token(R.t, R.n4, R.top_k + (R.shared ? 1 : 0))) sum_tokens_kernel<<<(unsigned)R.t, 256, 0, s>>>(R);
    else sum_sorted_kernel<<<(unsigned)((R.t * R.n4 + 255) / 256), 256, 0, s>>>(R);
    return cudaGetLastError();
}

// Expert-parallel dispatch packing: the routed rows of expert e (list `ids_map[e]`) go to positions
// [prefix(e), prefix(e) + tpe[e]) of the send buffers, as f16; experts are contiguous per destination rank,
// so the buffer is grouped by rank.  row_pos[flat id] remembers where each row went.
__global__ void __launch_bounds__(256) ep_pack_kernel(const float *__restrict__ x, const float *__restrict__ w,
                                                      const uint32_t *__restrict__ tpe, const int32_t *__restrict__ ids_map,
                                                      int map_stride, int top_k, int hidden, int e_local,
                                                      __half *__restrict__ rows, uint32_t *__restrict__ local_ids,
                                                      float *__restrict__ row_w, int32_t *__restrict__ row_pos) {
    __shared__ int warp_rows[8];
    __shared__ int row0_s;
    const int e = blockIdx.x;
    int rpart = 0;
    for (int i = threadIdx.x; i < e; i += 256) rpart += (int)tpe[i];
    for (int o = 16; o; o >>= 1) rpart += __shfl_xor_sync(0xffffffffu, rpart, o);
    if ((threadIdx.x & 31) == 0) warp_rows[threadIdx.x >> 5] = rpart;
    __syncthreads();
    if (threadIdx.x == 0) {
        int r = 0;
        for (int i = 0; i < 8; i++) r += warp_rows[i];
        row0_s = r;
    }
    __syncthreads();
    const int row0 = row0_s, n = (int)tpe[e], chunks = hidden / 8;
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        const int fid = ids_map[(size_t)e * map_stride + i];
        const int p = row0 + i;
        const float *src = x + (size_t)(fid / top_k) * hidden;
        __half *dst = rows + (size_t)p * hidden;
        for (int ci = threadIdx.x; ci < chunks; ci += 256) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(src) + 2 * ci);
            const float4 b = __ldg(reinterpret_cast<const float4 *>(src) + 2 * ci + 1);
            __align__(16) __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w),
                                          __floats2half2_rn(b.x, b.y), __floats2half2_rn(b.z, b.w)};
            reinterpret_cast<uint4 *>(dst)[ci] = *reinterpret_cast<const uint4 *>(h);
        }
        if (threadIdx.x == 0) {
            local_ids[p] = (uint32_t)(e % e_local);
            row_w[p] = w[fid];
            row_pos[fid] = p;
        }
    }
}

// send_counts[r] = rows routed to the experts of rank r
__global__ void ep_counts_kernel(const uint32_t *__restrict__ tpe, int n_expert, int e_local, long long *__restrict__ counts) {
    const int r = blockIdx.x;
    int c = 0;
    for (int e = r * e_local + threadIdx.x; e < (r + 1) * e_local && e < n_expert; e += 32) c += (int)tpe[e];
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (threadIdx.x == 0) counts[r] = c;
}

// identity row list for a one-expert stack: tpe[0] = t, ids_map[i] = i
__global__ void iota_list_kernel(int64_t t, uint32_t *tpe, int32_t *ids_map) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) tpe[0] = (uint32_t)t;
    if (i < t) ids_map[i] = (int32_t)i;
}

struct Carver {
    uint8_t *base;
    size_t off;
    template <typename T>
    T *take(size_t count) {
        T *p = reinterpret_cast<T *>(base + off);
        off += lmoe_align_up(count * sizeof(T), 256);
        return p;
    }
};

bool ffn_sorts(const lmoe_expert_stack *gate, const lmoe_expert_stack *up) { return gate->dtype == LMOE_Q4_K && up->dtype == LMOE_Q4_K; }

// The f16 activations of a grouped SwiGLU FFN: x_rows rows in token order for the fused gate/up kernel, else in tile order.
size_t ffn_x_bytes(const MmRows &R, int64_t x_rows, int64_t hidden, bool fused) {
    return fused ? lmoe_align_up((size_t)x_rows * hidden * 2, 256) : mm_tiled_bytes(R, hidden);
}
// Its scratch, by the form that `fused` takes.
size_t ffn_bytes(const MmRows &R, int64_t x_rows, int64_t hidden, int64_t ff, bool fused) {
    const size_t all = (size_t)(R.rows + R.extra);
    size_t o = 0;
    o += ffn_x_bytes(R, x_rows, hidden, fused);
    o += fused ? mm_src_bytes(R) : 0;                        // source row of every tile row
    o += lmoe_align_up(all * 4, 256);                        // position of every flat id
    o += (fused ? 1 : 2) * lmoe_align_up(all * ff * 4, 256); // SwiGLU activations, or gate and up
    o += mm_tiled_bytes(R, ff);                              // f16 activation in tile order
    o += lmoe_align_up(all * 4, 256);                        // row scale
    o += lmoe_align_up(all * 4, 256);                        // flat id of every sorted row
    o += mm_tiles_bytes(R);
    return o;
}

// y[rows, hidden] = row_weight * FFN_{expert of row}(x[row / top_k]); lists as produced by map0.
// With `spos` / `scale_out` (both [rows + extra], caller-owned) and Q4_K gate/up stacks, y instead holds the
// UNSCALED rows in expert-sorted order: row spos[flat id], to be multiplied by scale_out[that row]; the
// tensor-core epilogues then store whole tile columns side by side instead of scattering by flat id.  Only in that form
// can R.extra rows of the shared expert (`sh`: its gate, up, down) ride along: one launch of each kernel serves both.
// The lists must name every flat id, but for these: SLOTS_MAY_BE_EMPTY (sorted form), ids >= n_expert are empty slots;
// ROWS_MAY_BE_UNLISTED (unsorted), a row whose id is none of the experts' is a zero row.
enum Gaps { COMPLETE = 0, SLOTS_MAY_BE_EMPTY = 1, ROWS_MAY_BE_UNLISTED = 2 };

lmoe_status ffn_grouped(const MmRows &R, const lmoe_expert_stack *gate, const lmoe_expert_stack *up, const lmoe_expert_stack *down,
                        const lmoe_expert_stack *const (&sh)[3], const void *x, int top_k, const uint32_t *tpe, const int32_t *ids_map,
                        int64_t map_stride, const float *row_w, float *y, uint8_t *ws, uint32_t *flag, cudaStream_t s,
                        int32_t *spos = nullptr, float *scale_out = nullptr, int x_f16 = 0, int gaps = COMPLETE) {
    const int64_t all = R.rows + R.extra, ff = gate->n_out, hidden = gate->k;
    const bool fused_gu = ffn_sorts(gate, up), sorted = spos && scale_out && fused_gu;
    Carver c{ws, 0};
    uint8_t *xt = c.take<uint8_t>(ffn_x_bytes(R, R.rows / top_k, hidden, fused_gu));
    int32_t *src = reinterpret_cast<int32_t *>(c.take<uint8_t>(fused_gu ? mm_src_bytes(R) : 0));
    int32_t *pos = c.take<int32_t>((size_t)all);
    float *g = c.take<float>((size_t)all * ff), *u = c.take<float>(fused_gu ? 0 : (size_t)all * ff);
    uint8_t *act = c.take<uint8_t>(mm_tiled_bytes(R, ff));
    float *rs = c.take<float>((size_t)all);
    int32_t *sfid = c.take<int32_t>((size_t)all);
    void *tiles = ws + c.off;
    lmoe_status st;
    if (gaps == ROWS_MAY_BE_UNLISTED) LMOE_CUDA(cudaMemsetAsync(pos, 0xFF, (size_t)all * 4, s));
    if (gaps == SLOTS_MAY_BE_EMPTY) {
        // some (token, slot) pairs name no expert: the lists skip them, and the per-row arrays mark them
        if (!sorted) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "masked slots need the fused Q4_K gate/up kernel");
        LMOE_CUDA(cudaMemsetAsync(spos, 0xFF, (size_t)all * 4, s));
        LMOE_CUDA(cudaMemsetAsync(sfid, 0xFF, (size_t)all * 4, s));
    }
    const unsigned row_blocks = (unsigned)((all + 7) / 8);
    if (fused_gu) {
        // both projections in one pass over the activations, SwiGLU in the epilogue
        if ((st = launch_stage_rows(R, x, x_f16, R.rows / top_k, top_k, (int)hidden, tpe, ids_map, map_stride, tiles, xt, src, pos,
                                    sorted ? spos : nullptr, sorted ? sfid : nullptr, s)))
            return st;
        if ((st = launch_mm_gateup(R, gate, up, sh[0], sh[1], xt, src, ids_map, map_stride, g, sorted, tiles, flag, s))) return st;
        rescale_rows_kernel<<<row_blocks, 256, 0, s>>>(g, row_w, pos, sorted ? sfid : nullptr, all, R.rows, (int)ff, R.nt, act,
                                                       sorted ? scale_out : rs, y, (int)hidden);
        LMOE_LAUNCH_CHECK("rescale_rows_kernel");
    } else {
        if ((st = launch_gather_tiles(R, x, x_f16, 1, top_k, (int)hidden, tpe, ids_map, map_stride, tiles, xt, pos, nullptr, nullptr, s)))
            return st;
        if ((st = launch_mm_id(R, gate, nullptr, xt, ids_map, map_stride, nullptr, g, 0, tiles, flag, s))) return st;
        if ((st = launch_mm_id(R, up, nullptr, xt, ids_map, map_stride, nullptr, u, 0, tiles, flag, s))) return st;
        swiglu_rows_kernel<<<row_blocks, 256, 0, s>>>(g, u, row_w, pos, all, (int)ff, R.nt, act, rs, y, (int)hidden);
        LMOE_LAUNCH_CHECK("swiglu_rows_kernel");
    }
    return launch_mm_id(R, down, sh[2], act, ids_map, map_stride, sorted ? nullptr : rs, y, sorted, tiles, flag, s);
}

bool layer_mm_ok(const lmoe_layer *L) {
    return mm_id_kernel_available(L->gate->dtype, L->expert_ff, L->hidden) &&
           mm_id_kernel_available(L->down->dtype, L->hidden, L->expert_ff) && L->expert_ff % 256 == 0 &&
           L->hidden % 8 == 0;
}

} // namespace

// Scratch of the routed (+ shared) experts of `t` tokens with `top_k` slots each, after the routing decision.
static MmRows experts_rows(const lmoe_layer *L, int64_t t, int64_t top_k, int add_shared) {
    return mm_rows(t * top_k, add_shared && L->sh_gate && ffn_sorts(L->gate, L->up) ? t : 0, L->n_expert);
}
static size_t experts_ws_bytes(const lmoe_layer *L, int64_t t, int64_t top_k) {
    const MmRows R = experts_rows(L, t, top_k, 1);
    const size_t all = (size_t)(t * (top_k + 1));
    size_t o = 0;
    o += lmoe_map0_scratch_bytes(L->n_expert, t);
    o += lmoe_align_up(all * L->hidden * 4, 256);                    // partial rows
    o += lmoe_align_up((size_t)(t + 64) * 4, 256);                   // identity list
    o += 2 * lmoe_align_up(all * 4, 256);                            // sorted position and scale of every row
    const bool fused = ffn_sorts(L->gate, L->up);
    const size_t a = ffn_bytes(R, t, L->hidden, L->expert_ff, fused), b = ffn_bytes(mm_rows(t, 0, 1), t, L->hidden, L->expert_ff, fused);
    o += a > b ? a : b;
    return o;
}

// The experts of a block on a routing decision that is already on the device: per-expert row lists, grouped
// GEMMs, slot-order sum, optionally the shared expert and a residual.  x: [t, hidden] f32 or f16; ids / w: [t, top_k]
// (`masked`: ids >= n_expert are empty slots).  `ws` holds experts_ws_bytes(); `flag` is the device flag.
static lmoe_status experts_prefill(const lmoe_layer *L, const void *x, int x_f16, const uint32_t *ids, const float *w,
                                   int64_t t, int64_t top_k, int masked, int add_shared, const float *residual, float *out,
                                   uint8_t *ws, uint32_t *flag, cudaStream_t s) {
    const int64_t rows = t * top_k, H = L->hidden;
    const MmRows R = experts_rows(L, t, top_k, add_shared);
    Carver c{ws, 0};
    uint8_t *map0 = c.take<uint8_t>(lmoe_map0_scratch_bytes(L->n_expert, t));
    float *y = c.take<float>((size_t)(rows + t) * H);
    uint32_t *sh_list = c.take<uint32_t>((size_t)t + 64);
    int32_t *spos = c.take<int32_t>((size_t)(rows + t));
    float *rscale = c.take<float>((size_t)(rows + t));
    uint8_t *ffn_ws = ws + c.off;
    uint32_t *tpe = reinterpret_cast<uint32_t *>(map0);
    int32_t *ids_map = reinterpret_cast<int32_t *>(map0 + L->n_expert * 4);
    // ids >= n_expert match no expert's list: those slots stay empty
    LMOE_CUDA(launch_map0(ids, (int)t, (int)top_k, (int)L->n_expert, tpe, ids_map, s));
    const bool sorted = ffn_sorts(L->gate, L->up), shared = add_shared && L->sh_gate;
    lmoe_status st = ffn_grouped(R, L->gate, L->up, L->down, {R.extra ? L->sh_gate : nullptr, R.extra ? L->sh_up : nullptr, R.extra ? L->sh_down : nullptr},
                                 x, (int)top_k, tpe, ids_map, t, w, y, ffn_ws, flag, s, spos, rscale, x_f16, masked);
    if (st) return st;
    float *ysh = y + (size_t)rows * H;
    if (shared && !R.extra) {
        iota_list_kernel<<<(unsigned)((t + 255) / 256), 256, 0, s>>>(t, sh_list, reinterpret_cast<int32_t *>(sh_list + 64));
        LMOE_LAUNCH_CHECK("iota_list_kernel");
        st = ffn_grouped(mm_rows(t, 0, 1), L->sh_gate, L->sh_up, L->sh_down, {nullptr, nullptr, nullptr}, x, 1, sh_list,
                         reinterpret_cast<int32_t *>(sh_list + 64), t, nullptr, ysh, ffn_ws, flag, s, nullptr, nullptr, x_f16);
        if (st) return st;
    }
    const int64_t n = t * (H / 4);
    if (sorted)
        LMOE_CUDA(launch_sum_sorted({y, rscale, spos, shared ? y : nullptr, rscale, spos + rows, residual, t, (int)top_k, (int)(H / 4), out}, s));
    else
        sum_slots_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(y, shared ? ysh : nullptr, residual, t, (int)top_k, (int)(H / 4), out);
    LMOE_LAUNCH_CHECK("sum_slots_kernel");
    return LMOE_OK;
}

// Routing through route_filter.cu once the f32 product is the longer one.  A block's forward with experts of width 256, cold L2, us without / with:
//   tokens                    512          768         1024         2048         4096        16384
//   hidden 3072, 256     223 / 220    257 / 239    288 / 265    422 / 357    677 / 576   2290 / 1867
//   hidden 4096, 256     238 / 234    283 / 256    314 / 275    488 / 404    772 / 630   2599 / 2066
//   hidden 1024, 256         -        126 / 118    134 / 124    189 / 163    295 / 241    902 / 709
//   hidden 4096, 128     177 / 187    214 / 212    239 / 230    377 / 353    625 / 579   2115 / 1977
//   hidden 2048, 128         -        136 / 134    150 / 145    228 / 216    375 / 341   1197 / 1107
//   hidden 2048, 96          -            -        142 / 142    214 / 208    351 / 335   1138 / 1099
//   hidden 4096, 64          -        163 / 171    207 / 215    310 / 314    549 / 535   1880 / 1930
//   hidden 2304, 64          -            -            -        233 / 189    397 / 308   1374 / 1010
//   hidden 1280, 256         -        189 / 136    217 / 151    344 / 204    585 / 311   2079 / 961
// The tiled f32 product is for hidden a multiple of 512; without it the filter pays far sooner, and for 64 experts too.  Where the bounds tell next to nothing
// apart a call takes up to 4 to 25 % longer than without, see route_filter.cu, so the line lies where a plain prompt gains 4 %: 256 experts of 256, hidden 3072, 512 / 640 tokens
// 224 / 220 and 244 / 232 us, but with eight channels a hundred times the others 223 / 247 and 246 / 258.
static bool prefill_filters(const lmoe_layer *L, int64_t t) {
    const bool tiled = L->hidden % 512 == 0, early = !tiled || (L->hidden <= 2048 && L->n_expert >= 128);
    return (double)t * L->n_expert * L->hidden >= (early ? 3e8 : 5e8) && (!tiled || L->n_expert >= 96) && route_filter_available(L->hidden, L->n_expert, L->top_k);
}

// Scratch of the routing: the f32 logits, or the filter's, which has room for them (a call with unaligned operands takes the f32 routing all the same).
static size_t prefill_route_bytes(const lmoe_layer *L, int64_t t) {
    return prefill_filters(L, t) ? route_filter_bytes(t, L->hidden, L->n_expert) : (size_t)t * L->n_expert * 4;
}

size_t prefill_workspace_bytes(const lmoe_layer *L, int64_t t) {
    if (t < 1) t = 1;
    const int64_t rows = t * L->top_k;
    size_t o = 65536;
    o += lmoe_align_up(prefill_route_bytes(L, t), 256);
    o += 2 * lmoe_align_up((size_t)rows * 4, 256);                   // ids, weights
    o += experts_ws_bytes(L, t, L->top_k);
    return o;
}

lmoe_status launch_moe_prefill(const lmoe_layer *L, const float *x, const float *residual, int64_t t, float *out, uint32_t *ids_out,
                               float *w_out, void *workspace, size_t workspace_bytes, cudaStream_t s) {
    if (!layer_mm_ok(L)) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for this layer's shapes / dtypes");
    if (!workspace || workspace_bytes < prefill_workspace_bytes(L, t))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "prefill workspace needs %zu bytes, got %zu", prefill_workspace_bytes(L, t),
                         workspace_bytes);
    if (L->n_expert > 512) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "grouped GEMM supports at most 512 experts");
    if (t * L->top_k > INT32_MAX / 2) return lmoe_fail(LMOE_ERR_INVALID, "too many routed rows");
    const int64_t rows = t * L->top_k, H = L->hidden;
    Carver c{static_cast<uint8_t *>(workspace), 65536};
    uint32_t *flag = reinterpret_cast<uint32_t *>(workspace);
    uint8_t *route_ws = c.take<uint8_t>(prefill_route_bytes(L, t));
    uint32_t *ids = c.take<uint32_t>((size_t)rows);
    float *w = c.take<float>((size_t)rows);
    const bool filter = prefill_filters(L, t) && ((reinterpret_cast<uintptr_t>(L->router) | reinterpret_cast<uintptr_t>(x)) & 15u) == 0;
    uint8_t *ex_ws = static_cast<uint8_t *>(workspace) + c.off;

    // (both begin with a fresh device flag: the workspace needs no initialisation)
    if (filter) {
        LMOE_CUDA(launch_route_filter(L->router, L->bias, x, (int)t, (int)H, (int)L->n_expert, (int)L->top_k, L->scale, L->norm, route_ws, ids, w, flag, s));
    } else {
        float *logits = reinterpret_cast<float *>(route_ws);
        LMOE_CUDA(launch_route_logits(L->router, x, (int)t, (int)H, (int)L->n_expert, logits, s));
        LMOE_CUDA(launch_route_select(logits, L->bias, (int)t, (int)L->n_expert, (int)L->top_k, L->scale, L->norm, ids, w, s, flag));
    }
    lmoe_status st = experts_prefill(L, x, 0, ids, w, t, L->top_k, 0, 1, residual, out, ex_ws, flag, s);
    if (st) return st;
    if (ids_out) LMOE_CUDA(cudaMemcpyAsync(ids_out, ids, (size_t)rows * 4, cudaMemcpyDeviceToDevice, s));
    if (w_out) LMOE_CUDA(cudaMemcpyAsync(w_out, w, (size_t)rows * 4, cudaMemcpyDeviceToDevice, s));
    return LMOE_OK;
}

// `ExpertFfn::forward` on the grouped-GEMM path (see lmoe_experts_forward): the caller's routing decision.
size_t experts_prefill_workspace_bytes(const lmoe_layer *L, int64_t t) {
    return 65536 + experts_ws_bytes(L, t < 1 ? 1 : t, L->top_k);
}
lmoe_status launch_experts_prefill(const lmoe_layer *L, const float *x, const uint32_t *ids, const float *w, int64_t t,
                                   int add_shared, float *out, void *workspace, size_t workspace_bytes, cudaStream_t s) {
    if (!layer_mm_ok(L)) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for this layer's shapes / dtypes");
    if (!workspace || workspace_bytes < experts_prefill_workspace_bytes(L, t))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "workspace needs %zu bytes, got %zu", experts_prefill_workspace_bytes(L, t),
                         workspace_bytes);
    if (t * L->top_k > INT32_MAX / 2) return lmoe_fail(LMOE_ERR_INVALID, "too many routed rows");
    uint32_t *flag = reinterpret_cast<uint32_t *>(workspace);
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    return experts_prefill(L, x, 0, ids, w, t, L->top_k, 1, add_shared, nullptr, out, static_cast<uint8_t *>(workspace) + 65536, flag, s);
}

// ---- op-level entry points ------------------------------------------------------------
extern "C" int32_t lmoe_mm_id_supported(int32_t dtype, int64_t top_k) {
    return (dtype == LMOE_Q4_K || dtype == LMOE_Q6_K) && top_k >= 1 ? 1 : 0;
}

extern "C" size_t lmoe_mm_id_workspace_bytes(const lmoe_expert_stack *stack, int64_t t, int64_t top_k, int64_t x_per_row) {
    if (!stack || t < 0 || top_k < 1 || x_per_row < 1) return 0;
    const MmRows R = mm_rows(t * top_k, 0, stack->n_expert);
    return 256 + mm_tiled_bytes(R, stack->k) + mm_tiles_bytes(R);
}

static lmoe_status mm_id_run(const lmoe_expert_stack *stack, const float *x, int64_t t, int64_t x_per_row, int64_t k,
                             const uint32_t *ids, int64_t t_ids, int64_t top_k, const void *map0, float *out,
                             void *workspace, size_t workspace_bytes, cudaStream_t s) {
    lmoe_status st = lmoe_id_shape_check(stack, x, t, x_per_row, k, ids, t_ids, top_k, out);
    if (st) return st;
    if (!mm_id_kernel_available(stack->dtype, stack->n_out, stack->k))
        return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for dtype %d, n_out %lld, k %lld", stack->dtype,
                         (long long)stack->n_out, (long long)stack->k);
    const size_t need = lmoe_mm_id_workspace_bytes(stack, t, top_k, x_per_row);
    if (!workspace || workspace_bytes < need)
        return lmoe_fail(LMOE_ERR_WORKSPACE, "mul_mm_id workspace needs %zu bytes, got %zu", need, workspace_bytes);
    if (t == 0) return LMOE_OK;
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    uint32_t *flag = reinterpret_cast<uint32_t *>(ws);
    uint8_t *xt = ws + 256;
    const MmRows R = mm_rows(t * top_k, 0, stack->n_expert);
    void *tiles = ws + 256 + mm_tiled_bytes(R, k);
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    const uint32_t *tpe = static_cast<const uint32_t *>(map0);
    const int32_t *ids_map = reinterpret_cast<const int32_t *>(static_cast<const uint8_t *>(map0) + stack->n_expert * 4);
    if ((st = launch_gather_tiles(R, x, 0, (int)x_per_row, (int)top_k, (int)k, tpe, ids_map, t, tiles, xt, nullptr, nullptr, nullptr, s)))
        return st;
    return launch_mm_id(R, stack, nullptr, xt, ids_map, t, nullptr, out, 0, tiles, flag, s);
}

extern "C" lmoe_status lmoe_mul_mm_id_shared(const lmoe_expert_stack *stack, const float *x, int64_t t, int64_t x_per_row,
                                             int64_t k, const uint32_t *ids, int64_t t_ids, int64_t top_k,
                                             const void *map0_scratch, int64_t map_n_expert, int64_t map_t,
                                             int64_t map_top_k, float *out, void *workspace, size_t workspace_bytes,
                                             void *stream) {
    lmoe_clear_error();
    if (!stack) return lmoe_fail(LMOE_ERR_INVALID, "expert stack is NULL");
    if (!map0_scratch) return lmoe_fail(LMOE_ERR_INVALID, "map0 scratch is NULL");
    // the consumer re-validates the producer's geometry, src/ops/dispatch.rs:903-909
    if (map_n_expert != stack->n_expert || map_t != t || map_top_k != top_k)
        return lmoe_fail(LMOE_ERR_INVALID,
                         "shared map0 scratch geometry (n_expert=%lld, t=%lld, top_k=%lld) does not match this projection "
                         "(n_expert=%lld, t=%lld, top_k=%lld); the ids-map offset would be wrong",
                         (long long)map_n_expert, (long long)map_t, (long long)map_top_k, (long long)stack->n_expert,
                         (long long)t, (long long)top_k);
    return mm_id_run(stack, x, t, x_per_row, k, ids, t_ids, top_k, map0_scratch, out, workspace, workspace_bytes,
                     (cudaStream_t)stream);
}

extern "C" lmoe_status lmoe_mul_mm_id(const lmoe_expert_stack *stack, const float *x, int64_t t, int64_t x_per_row,
                                      int64_t k, const uint32_t *ids, int64_t t_ids, int64_t top_k, float *out,
                                      void *workspace, size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    if (!stack) return lmoe_fail(LMOE_ERR_INVALID, "expert stack is NULL");
    lmoe_status st = lmoe_id_shape_check(stack, x, t, x_per_row, k, ids, t_ids, top_k, out);
    if (st) return st;
    const size_t mm = lmoe_mm_id_workspace_bytes(stack, t, top_k, x_per_row), mp = lmoe_map0_scratch_bytes(stack->n_expert, t);
    if (!workspace || workspace_bytes < mm + mp)
        return lmoe_fail(LMOE_ERR_WORKSPACE, "mul_mm_id workspace needs %zu bytes, got %zu", mm + mp, workspace_bytes);
    uint8_t *map0 = static_cast<uint8_t *>(workspace) + mm;
    LMOE_CUDA(launch_map0(ids, (int)t, (int)top_k, (int)stack->n_expert, reinterpret_cast<uint32_t *>(map0),
                          reinterpret_cast<int32_t *>(map0 + stack->n_expert * 4), (cudaStream_t)stream));
    return mm_id_run(stack, x, t, x_per_row, k, ids, t_ids, top_k, map0, out, workspace, mm, (cudaStream_t)stream);
}

// The grouped-GEMM branch of `FusedExperts::forward` as one call: map0, mul_mm_id (gate, up), silu_mul, l2_rescale, mul_mm_id
// (down), combine, with the bits of the ops one by one.  The tables and the f16 copy of x are made once for both projections,
// and the activations go straight into the down product's operand.
struct FfnMmLayout {
    MmRows R;
    size_t map0, tiles, xt, pos, g, u, act, l2, d, total;
    FfnMmLayout(const lmoe_expert_stack *gate, const lmoe_expert_stack *down, int64_t t, int64_t top_k) : R(mm_rows(t * top_k, 0, gate->n_expert)) {
        const size_t rows = (size_t)R.rows;
        size_t o = 256; // device flag
        auto take = [&](size_t n) { const size_t at = o; o += lmoe_align_up(n, 256); return at; };
        map0 = take(lmoe_map0_scratch_bytes(gate->n_expert, t));
        tiles = take(mm_tiles_bytes(R));
        xt = take(mm_tiled_bytes(R, gate->k));
        pos = take(rows * 4);
        g = take(rows * gate->n_out * 4);
        u = take(rows * gate->n_out * 4);
        act = take(mm_tiled_bytes(R, gate->n_out));
        l2 = take(rows * 4);
        d = take(rows * down->n_out * 4);
        total = o;
    }
};

extern "C" size_t lmoe_ffn_mm_workspace_bytes(const lmoe_expert_stack *gate, const lmoe_expert_stack *down, int64_t t, int64_t top_k) {
    if (!gate || !down || t < 0 || top_k < 1 || t * top_k > INT32_MAX / 2) return 0;
    return FfnMmLayout(gate, down, t, top_k).total;
}

extern "C" lmoe_status lmoe_ffn_mm(const lmoe_expert_stack *gate, const lmoe_expert_stack *up, const lmoe_expert_stack *down, const uint32_t *ids,
                                   int64_t t_ids, int64_t top_k, const float *weights, const float *x, int64_t t, int64_t k, float *out,
                                   void *workspace, size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    cudaStream_t s = (cudaStream_t)stream;
    if (!gate || !up || !down || !weights) return lmoe_fail(LMOE_ERR_INVALID, "an expert stack or the weights are NULL");
    lmoe_status st;
    if ((st = lmoe_id_shape_check(gate, x, t, 1, k, ids, t_ids, top_k, out)) || (st = lmoe_id_shape_check(up, x, t, 1, k, ids, t_ids, top_k, out)) ||
        (st = lmoe_id_shape_check(down, x, t, top_k, gate->n_out, ids, t_ids, top_k, out)) || (st = lmoe_combine_check(t, top_k, down->n_out)))
        return st;
    if (gate->n_out != up->n_out || gate->n_expert != up->n_expert || gate->n_expert != down->n_expert)
        return lmoe_fail(LMOE_ERR_INVALID, "the stacks disagree: gate %lld x %lld, up %lld x %lld, down %lld experts", (long long)gate->n_expert,
                         (long long)gate->n_out, (long long)up->n_expert, (long long)up->n_out, (long long)down->n_expert);
    for (const lmoe_expert_stack *e : {gate, up, down})
        if (!mm_id_kernel_available(e->dtype, e->n_out, e->k))
            return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for dtype %d, n_out %lld, k %lld", e->dtype, (long long)e->n_out,
                             (long long)e->k);
    if (t * top_k > INT32_MAX / 2 || t * top_k * gate->n_out > INT32_MAX)
        return lmoe_fail(LMOE_ERR_INVALID, "silu_mul n (%lld) must be in [0, i32::MAX]", (long long)(t * top_k * gate->n_out));
    if (gate->n_out > LMOE_FFN_MM_MAX_FF) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "expert width %lld: call the ops one by one", (long long)gate->n_out);
    const FfnMmLayout L(gate, down, t, top_k);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255u) || workspace_bytes < L.total)
        return lmoe_fail(LMOE_ERR_WORKSPACE, "ffn_mm workspace needs %zu bytes, 256-byte aligned, got %zu", L.total, workspace_bytes);
    if (t == 0) return LMOE_OK;
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    uint32_t *flag = reinterpret_cast<uint32_t *>(ws), *tpe = reinterpret_cast<uint32_t *>(ws + L.map0);
    int32_t *ids_map = reinterpret_cast<int32_t *>(ws + L.map0 + gate->n_expert * 4), *pos = reinterpret_cast<int32_t *>(ws + L.pos);
    float *g = reinterpret_cast<float *>(ws + L.g), *u = reinterpret_cast<float *>(ws + L.u), *l2 = reinterpret_cast<float *>(ws + L.l2);
    float *d = reinterpret_cast<float *>(ws + L.d);
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    LMOE_CUDA(cudaMemsetAsync(pos, 0xFF, (size_t)L.R.rows * 4, s)); // an id that names no expert
    LMOE_CUDA(launch_map0(ids, (int)t, (int)top_k, (int)gate->n_expert, tpe, ids_map, s));
    if ((st = launch_gather_tiles(L.R, x, 0, 1, (int)top_k, (int)k, tpe, ids_map, t, ws + L.tiles, ws + L.xt, pos, nullptr, nullptr, s))) return st;
    if ((st = launch_mm_id(L.R, gate, nullptr, ws + L.xt, ids_map, t, nullptr, g, 0, ws + L.tiles, flag, s))) return st;
    if ((st = launch_mm_id(L.R, up, nullptr, ws + L.xt, ids_map, t, nullptr, u, 0, ws + L.tiles, flag, s))) return st;
    LMOE_CUDA(launch_silu_rescale_tiles(g, u, pos, L.R.rows, (int)gate->n_out, L.R.nt, ws + L.act, l2, d, (int)down->n_out, s));
    if ((st = launch_mm_id(L.R, down, nullptr, ws + L.act, ids_map, t, nullptr, d, 0, ws + L.tiles, flag, s))) return st;
    LMOE_CUDA(launch_combine(d, l2, weights, (int)t, (int)top_k, (int)down->n_out, out, s, flag));
    return LMOE_OK;
}

// ---- expert-parallel pieces -------------------------------------------------------------
// (the same entries serve the shared expert alone, whose single list may take another tile size)
static size_t rows_ffn_bytes(const lmoe_layer *L, int64_t rows) {
    const bool fused = ffn_sorts(L->gate, L->up);
    const size_t a = ffn_bytes(mm_rows(rows, 0, L->n_expert), rows, L->hidden, L->expert_ff, fused);
    const size_t b = ffn_bytes(mm_rows(rows, 0, 1), rows, L->hidden, L->expert_ff, fused);
    return a > b ? a : b;
}
static size_t rows_ws_bytes(const lmoe_layer *L, int64_t rows) {
    return 65536 + lmoe_map0_scratch_bytes(L->n_expert, rows) + lmoe_align_up((size_t)(rows + 64) * 4, 256) +
           rows_ffn_bytes(L, rows);
}

static lmoe_status experts_rows_run(const lmoe_layer *L, const void *x, int x_f16, const uint32_t *local_ids,
                                    const float *row_weights, int64_t rows, float *out, void *workspace,
                                    size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    if (!L || !x || !local_ids || !out) return lmoe_fail(LMOE_ERR_INVALID, "layer/x/local_ids/out is NULL");
    if (rows < 0 || rows > INT32_MAX / 2) return lmoe_fail(LMOE_ERR_INVALID, "rows out of range");
    if (rows == 0) return LMOE_OK;
    if (reinterpret_cast<uintptr_t>(x) & 15u) return lmoe_fail(LMOE_ERR_INVALID, "x must be 16-byte aligned");
    if (!layer_mm_ok(L)) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for this layer's shapes / dtypes");
    if (!workspace || workspace_bytes < rows_ws_bytes(L, rows))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "workspace needs %zu bytes, got %zu", rows_ws_bytes(L, rows), workspace_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    Carver c{static_cast<uint8_t *>(workspace), 65536};
    uint32_t *flag = reinterpret_cast<uint32_t *>(workspace);
    uint8_t *map0 = c.take<uint8_t>(lmoe_map0_scratch_bytes(L->n_expert, rows));
    uint8_t *ffn_ws = static_cast<uint8_t *>(workspace) + c.off;
    uint32_t *tpe = reinterpret_cast<uint32_t *>(map0);
    int32_t *ids_map = reinterpret_cast<int32_t *>(map0 + L->n_expert * 4);
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    LMOE_CUDA(launch_map0(local_ids, (int)rows, 1, (int)L->n_expert, tpe, ids_map, s));
    return ffn_grouped(mm_rows(rows, 0, L->n_expert), L->gate, L->up, L->down, {nullptr, nullptr, nullptr}, x, 1, tpe, ids_map, rows,
                       row_weights, out, ffn_ws, flag, s, nullptr, nullptr, x_f16, ROWS_MAY_BE_UNLISTED);
}

extern "C" lmoe_status lmoe_experts_forward_rows(const lmoe_layer *L, const float *x, const uint32_t *local_ids,
                                                 const float *row_weights, int64_t rows, float *out, void *workspace,
                                                 size_t workspace_bytes, void *stream) {
    return experts_rows_run(L, x, 0, local_ids, row_weights, rows, out, workspace, workspace_bytes, stream);
}

extern "C" lmoe_status lmoe_experts_forward_rows_f16(const lmoe_layer *L, const void *x_f16, const uint32_t *local_ids,
                                                     const float *row_weights, int64_t rows, float *out, void *workspace,
                                                     size_t workspace_bytes, void *stream) {
    return experts_rows_run(L, x_f16, 1, local_ids, row_weights, rows, out, workspace, workspace_bytes, stream);
}

// Token-level form for the expert-parallel exchange: one activation row per token, up to top_k experts each.
static size_t tokens_ws_bytes(const lmoe_layer *L, int64_t t, int64_t top_k) {
    return 65536 + experts_ws_bytes(L, t, top_k);
}

extern "C" size_t lmoe_tokens_workspace_bytes(const lmoe_layer *L, int64_t t, int64_t top_k) {
    return L && top_k >= 1 ? tokens_ws_bytes(L, t < 1 ? 1 : t, top_k) : 0;
}

extern "C" lmoe_status lmoe_experts_forward_tokens_f16(const lmoe_layer *L, const void *x_f16, const uint32_t *ids,
                                                       const float *weights, int64_t t, int64_t top_k, float *out,
                                                       void *workspace, size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    if (!L || !x_f16 || !ids || !weights || !out) return lmoe_fail(LMOE_ERR_INVALID, "layer/x/ids/weights/out is NULL");
    if (top_k < 1 || t < 0 || t * top_k > INT32_MAX / 2) return lmoe_fail(LMOE_ERR_INVALID, "t / top_k out of range");
    if (t == 0) return LMOE_OK;
    if ((reinterpret_cast<uintptr_t>(x_f16) | reinterpret_cast<uintptr_t>(out)) & 15u)
        return lmoe_fail(LMOE_ERR_INVALID, "x and out must be 16-byte aligned");
    if (!layer_mm_ok(L)) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for this layer's shapes / dtypes");
    if (!workspace || workspace_bytes < tokens_ws_bytes(L, t, top_k))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "workspace needs %zu bytes, got %zu", tokens_ws_bytes(L, t, top_k), workspace_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t *flag = reinterpret_cast<uint32_t *>(workspace);
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    return experts_prefill(L, x_f16, 1, ids, weights, t, top_k, 1, 0, nullptr, out, static_cast<uint8_t *>(workspace) + 65536, flag, s);
}

extern "C" lmoe_status lmoe_shared_forward(const lmoe_layer *L, const float *x, int64_t t, float *out, void *workspace,
                                           size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    if (!L || !x || !out) return lmoe_fail(LMOE_ERR_INVALID, "layer/x/out is NULL");
    if (!L->sh_gate) return lmoe_fail(LMOE_ERR_INVALID, "the layer has no shared expert");
    if (t < 0 || t > INT32_MAX / 2) return lmoe_fail(LMOE_ERR_INVALID, "t out of range");
    if (t == 0) return LMOE_OK;
    if (!layer_mm_ok(L)) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "no grouped-GEMM kernel for this layer's shapes / dtypes");
    if (!workspace || workspace_bytes < rows_ws_bytes(L, t))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "workspace needs %zu bytes, got %zu", rows_ws_bytes(L, t), workspace_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    Carver c{static_cast<uint8_t *>(workspace), 65536};
    uint32_t *flag = reinterpret_cast<uint32_t *>(workspace);
    uint32_t *list = c.take<uint32_t>((size_t)t + 64);
    uint8_t *ffn_ws = static_cast<uint8_t *>(workspace) + c.off;
    LMOE_CUDA(cudaMemsetAsync(flag, 0, 16, s));
    iota_list_kernel<<<(unsigned)((t + 255) / 256), 256, 0, s>>>(t, list, reinterpret_cast<int32_t *>(list + 64));
    LMOE_LAUNCH_CHECK("iota_list_kernel");
    return ffn_grouped(mm_rows(t, 0, 1), L->sh_gate, L->sh_up, L->sh_down, {nullptr, nullptr, nullptr}, x, 1, list,
                       reinterpret_cast<int32_t *>(list + 64), t, nullptr, out, ffn_ws, flag, s);
}

extern "C" size_t lmoe_rows_workspace_bytes(const lmoe_layer *L, int64_t rows) {
    return L ? rows_ws_bytes(L, rows < 1 ? 1 : rows) : 0;
}

// Expert-parallel exchange helpers (no counterpart in the single-GPU reference).
extern "C" size_t lmoe_ep_pack_workspace_bytes(int64_t n_expert, int64_t t) { return lmoe_map0_scratch_bytes(n_expert, t); }

extern "C" lmoe_status lmoe_ep_pack(const float *x, const uint32_t *ids, const float *weights, int64_t t, int64_t hidden,
                                    int64_t top_k, int64_t n_expert, int64_t world, void *rows_f16, uint32_t *local_ids,
                                    float *row_weights, int32_t *row_pos, int64_t *send_counts, void *workspace,
                                    size_t workspace_bytes, void *stream) {
    lmoe_clear_error();
    if (!x || !ids || !weights || !rows_f16 || !local_ids || !row_weights || !row_pos || !send_counts)
        return lmoe_fail(LMOE_ERR_INVALID, "ep_pack: a buffer is NULL");
    if (t < 0 || top_k < 1 || n_expert < 1 || world < 1 || n_expert % world || hidden < 8 || hidden % 8)
        return lmoe_fail(LMOE_ERR_INVALID, "ep_pack: t >= 0, top_k >= 1, n_expert divisible by world, hidden a multiple of 8 required");
    if (t * top_k > INT32_MAX / 2 || n_expert > 65535) return lmoe_fail(LMOE_ERR_INVALID, "ep_pack: problem too large");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(rows_f16)) & 15u)
        return lmoe_fail(LMOE_ERR_INVALID, "ep_pack: x and rows_f16 must be 16-byte aligned");
    if (!workspace || workspace_bytes < lmoe_map0_scratch_bytes(n_expert, t))
        return lmoe_fail(LMOE_ERR_WORKSPACE, "ep_pack workspace needs %zu bytes, got %zu", lmoe_map0_scratch_bytes(n_expert, t),
                         workspace_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t *tpe = static_cast<uint32_t *>(workspace);
    int32_t *ids_map = reinterpret_cast<int32_t *>(static_cast<uint8_t *>(workspace) + n_expert * 4);
    LMOE_CUDA(cudaMemsetAsync(row_pos, 0xFF, (size_t)(t * top_k) * 4, s)); // an id that names no expert: an empty slot
    LMOE_CUDA(launch_map0(ids, (int)t, (int)top_k, (int)n_expert, tpe, ids_map, s));
    const int e_local = (int)(n_expert / world);
    ep_counts_kernel<<<(unsigned)world, 32, 0, s>>>(tpe, (int)n_expert, e_local, reinterpret_cast<long long *>(send_counts));
    LMOE_LAUNCH_CHECK("ep_counts_kernel");
    if (t > 0) {
        const int gy = n_expert >= 64 ? 16 : (n_expert >= 8 ? 128 : 1024);
        ep_pack_kernel<<<dim3((unsigned)n_expert, gy), 256, 0, s>>>(x, weights, tpe, ids_map, (int)t, (int)top_k, (int)hidden, e_local,
                                                                static_cast<__half *>(rows_f16), local_ids, row_weights, row_pos);
        LMOE_LAUNCH_CHECK("ep_pack_kernel");
    }
    return LMOE_OK;
}

extern "C" lmoe_status lmoe_ep_localize_ids(const uint32_t *ids, int64_t n, int64_t first, int64_t count, uint32_t *out,
                                            void *stream) {
    lmoe_clear_error();
    if (!ids || !out) return lmoe_fail(LMOE_ERR_INVALID, "ep_localize_ids: ids/out is NULL");
    if (n < 0 || first < 0 || count < 1 || first + count > (int64_t)UINT32_MAX)
        return lmoe_fail(LMOE_ERR_INVALID, "ep_localize_ids: n >= 0, first >= 0, count >= 1 required");
    LMOE_CUDA(launch_ep_localize_ids(ids, n, (uint32_t)first, (uint32_t)count, out, (cudaStream_t)stream));
    return LMOE_OK;
}

extern "C" lmoe_status lmoe_ep_combine(const float *rows, const int32_t *row_pos, const float *shared, int64_t t,
                                       int64_t top_k, int64_t hidden, float *out, void *stream) {
    lmoe_clear_error();
    if (!rows || !row_pos || !out) return lmoe_fail(LMOE_ERR_INVALID, "ep_combine: rows/row_pos/out is NULL");
    if (t < 0 || top_k < 1 || hidden < 4 || hidden % 4) return lmoe_fail(LMOE_ERR_INVALID, "ep_combine: bad dimensions");
    if ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(shared)) & 15u)
        return lmoe_fail(LMOE_ERR_INVALID, "ep_combine: rows, shared and out must be 16-byte aligned");
    if (t == 0) return LMOE_OK;
    LMOE_CUDA(launch_sum_sorted({rows, nullptr, row_pos, shared, nullptr, nullptr, nullptr, t, (int)top_k, (int)(hidden / 4), out}, (cudaStream_t)stream));
    return LMOE_OK;
}
