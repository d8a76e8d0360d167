// Grouped (indexed) quantized GEMM on the 5th-generation tensor cores: for every
// expert e, the rows routed to e times W[e]^T, scattered back to [t, top_k, n_out].
//
// Reference: `ops::mul_mm_id{,_shared}`, src/ops/mm_id.rs:16-39 ->
// kernel_mul_mm_id_q{4,6}_K_f32_t, src/ops/mm_id.metal:492-647 (f16 operand
// tiles, f32 accumulation); per-expert lists from map0, src/ops/mm_id.metal:207-269.
//
// Persistent pairs of CTAs, one CTA per SM, warp-specialised around tcgen05.mma; see grouped_mm_kernel.  The weight tile is the
// A operand (M = 256 output features, 128 in each CTA) and the routed rows are the N dimension, so ragged per-expert row counts cost
// only a rounding to 16.  Every wait is bounded; a wait that runs out records a flag and the kernel drains and exits.
#include <type_traits>

#include <cuda.h> // CUtensorMap (types only; the encoder is fetched through the runtime)

#include "fused.cuh"
#include "kquant.cuh"
#include "tc.cuh"

namespace {

constexpr int MM_M = 128;      // weight rows per CTA; a pair's tile has twice as many
// CG below: the CTAs that share a tile, 2 (a pair) or 1
constexpr int MM_K = 64;       // k per pipeline stage (one 128-byte swizzle row of f16)

// ---- PTX helpers ---------------------------------------------------------------
// Arrival at a barrier of the pair's first CTA.  Of the default scope: it may announce what lies in tensor memory, behind the tcgen05
// fence, or in this CTA's own shared memory, behind a proxy fence or a bulk copy's completion; nothing else that the other CTA reads.
template <int CG>
__device__ __forceinline__ void mb_arrive_first(uint64_t *b) {
    if (CG == 1) return mb_arrive(b);
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
                 "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(s32(b)) : "memory");
}
__device__ __noinline__ void mm_timeout(uint32_t *flag, uint32_t where) {
    if (atomicCAS(flag, 0u, (uint32_t)LMOE_FLAG_WAIT_TIMEOUT) == 0u) {
        flag[1] = 0x1000u + where;
        flag[2] = blockIdx.x;
    }
}
// 2-D tiled TMA load global -> shared (x = byte offset inside the row, a multiple of 16; y = row).
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     s32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(s32(bar))
                 : "memory");
}
// D += A * B for both CTAs of a pair; the A operand lies in tensor memory, in each CTA its own 128 lanes (weight rows) x 8 columns
// (K = 16 as f16 pairs), and each CTA's shared memory holds half of B's rows at the place the descriptor names.
// The four K = 16 steps of a 64-k block, of one projection or (d1 != d0) two: one piece of assembly of 32-bit additions, as the issuing
// warp's own instructions are what a thin tile's stage takes.  `first`: the block starts the accumulators.
template <int CG, bool TWO>
__device__ __forceinline__ void tc_mma_block(uint32_t d0, uint32_t d1, uint32_t a, uint32_t blo, uint32_t bhi, uint32_t idesc, uint32_t first) {
    if (CG == 1 && !TWO)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t.reg .b32 l, t;\n\tsetp.eq.b32 p, %6, 0;\n\t"
                     "mov.b64 b, {%3, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%2], b, %5, p;\n\t"
                     "add.u32 l, %3, 2;\n\tadd.u32 t, %2, 8;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 4;\n\tadd.u32 t, %2, 16;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 6;\n\tadd.u32 t, %2, 24;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [t], b, %5, 1;\n\t}"
                     ::"r"(d0), "r"(d1), "r"(a), "r"(blo), "r"(bhi), "r"(idesc), "r"(first) : "memory");
    else if (CG == 2 && !TWO)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t.reg .b32 l, t;\n\tsetp.eq.b32 p, %6, 0;\n\t"
                     "mov.b64 b, {%3, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%2], b, %5, p;\n\t"
                     "add.u32 l, %3, 2;\n\tadd.u32 t, %2, 8;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 4;\n\tadd.u32 t, %2, 16;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 6;\n\tadd.u32 t, %2, 24;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t}"
                     ::"r"(d0), "r"(d1), "r"(a), "r"(blo), "r"(bhi), "r"(idesc), "r"(first) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t.reg .b32 l, t;\n\tsetp.eq.b32 p, %6, 0;\n\t"
                     "mov.b64 b, {%3, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%2], b, %5, p;\n\t"
                     "add.u32 t, %2, 32;\n\ttcgen05.mma.cta_group::2.kind::f16 [%1], [t], b, %5, p;\n\t"
                     "add.u32 l, %3, 2;\n\tadd.u32 t, %2, 8;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 t, %2, 40;\n\ttcgen05.mma.cta_group::2.kind::f16 [%1], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 4;\n\tadd.u32 t, %2, 16;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 t, %2, 48;\n\ttcgen05.mma.cta_group::2.kind::f16 [%1], [t], b, %5, 1;\n\t"
                     "add.u32 l, %3, 6;\n\tadd.u32 t, %2, 24;\n\tmov.b64 b, {l, %4};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [t], b, %5, 1;\n\t"
                     "add.u32 t, %2, 56;\n\ttcgen05.mma.cta_group::2.kind::f16 [%1], [t], b, %5, 1;\n\t}"
                     ::"r"(d0), "r"(d1), "r"(a), "r"(blo), "r"(bhi), "r"(idesc), "r"(first) : "memory");
}
// 32 registers of every lane -> 32 columns of the warp's 32 tensor-memory lanes; complete after tc_wait_st().
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
        "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
        "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 8 registers of every lane -> 8 columns of the warp's 32 tensor-memory lanes
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// ---- dequantisation ----------------------------------------------------------------
// The conversion is bound by instruction issue, so every operation is one instruction by construction.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// (base + a | base + b) - base, times scale, minus bias: exact integers in f16, one rounding in the fma
__device__ __forceinline__ uint32_t h2_sub_fma(uint32_t v, uint32_t base, uint32_t s, uint32_t m) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tsub.rn.f16x2 t, %1, %2;\n\tfma.rn.f16x2 %0, t, %3, %4;\n\t}" : "=r"(r) : "r"(v), "r"(base), "r"(s), "r"(m));
    return r;
}
__device__ __forceinline__ uint32_t h2_sub_mul(uint32_t v, uint32_t base, uint32_t s) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tsub.rn.f16x2 t, %1, %2;\n\tmul.rn.f16x2 %0, t, %3;\n\t}" : "=r"(r) : "r"(v), "r"(base), "r"(s));
    return r;
}

// ---- row tiles -----------------------------------------------------------------------
// The routed rows of an expert are cut into as few tiles as nt rows each allow, of even height: sixteens of rows, a tile one
// more or less than another.  A stage of a tile takes the multiplies' time, but from about 150 rows down the conversion's, which
// is the same for any height, so a full tile and a thin one cost more than two even ones (256 experts, 8192 tokens 2383 us
// with full tiles and a rest, 2348 so; Zipf, 6000 tokens 1935 and 1888).  tiles[i] = {expert, first list index,
// valid rows, first row in expert-sorted order}; i is also the slot of the tile in the tile-ordered operands.  A GEMM tile is (row
// tile, block of CG x 128 weight rows), the latter varying fastest, so CTAs running side by side share the same activation rows in L2.
// With `extra` > 0 one more list follows the experts' ("expert" n_expert): the rows 0 .. extra-1 of the shared expert.
// The tiles stand by falling height: the CTAs take the tiles of a product in turn, so each round has tiles of one cost and the
// last, incomplete one the cheapest (experts' order left the SMs idle for 13 % of the gate/up product of 2048 tokens; the whole
// call 920 -> 892 us, 600 tokens with 128 experts of 768 217 -> 208).
__global__ void __launch_bounds__(1024) row_tiles_kernel(const uint32_t *__restrict__ tpe, int n_expert, int extra, int nt,
                                                         int4 *__restrict__ tiles, int32_t *__restrict__ n_tiles, int max_tiles) {
    pdl_begin();
    __shared__ int warp_sum[32];
    __shared__ int2 of_height[1024];  // an expert's tiles of its larger and its smaller height: height << 24 | count
    __shared__ int first[32][16];     // tiles by warp and height, then the place of the first of them
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    const int rows = e < n_expert ? (int)tpe[e] : (e == n_expert ? extra : 0);
    const int n16 = (rows + 15) / 16, n = (rows + nt - 1) / nt, low = n ? n16 / n : 0, high_n = n ? n16 - low * n : 0;
    int cr = rows; // inclusive prefix sum
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, cr, o);
        if (lane >= o) cr += v;
    }
    if (lane == 31) warp_sum[warp] = cr;
    // the warp's tiles by height, and how many of a lane's height are before its own
    int at_high = 0, at_low;
    if (lane < 16) first[warp][lane] = 0;
    __syncwarp();
    if (!__any_sync(0xffffffffu, n > 1)) { // one tile each
        const uint32_t same = __match_any_sync(0xffffffffu, low);
        at_low = __popc(same & ((1u << lane) - 1u));
        if (at_low == 0) first[warp][low] = __popc(same);
    } else { // the larger heights first, then the smaller ones
        of_height[e] = make_int2((low + 1) << 24 | high_n, low << 24 | (n - high_n)); // a list has fewer than 2^24 tiles
        __syncwarp();
        int all = 0;
        at_low = 0;
        for (uint32_t left = __ballot_sync(0xffffffffu, n > 0); left; left &= left - 1u) {
            const int l = __ffs(left) - 1;
            const int2 h = of_height[32 * warp + l];
            const int hh = h.x >> 24, hn = h.x & 0xffffff, lh = h.y >> 24, ln = h.y & 0xffffff;
            all += (hh == lane ? hn : 0) + (lh == lane ? ln : 0);
            at_high += l < lane && hh == low + 1 ? hn : 0;
            at_low += (hh == low ? hn : 0) + (l < lane && lh == low ? ln : 0);
        }
        if (lane < 16) first[warp][lane] = all;
    }
    __syncthreads();
    if (warp == 0) {
        int v = warp_sum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += a;
        }
        warp_sum[lane] = v;
    } else if (warp == 1 && lane < 16) { // the warps' counts of a height -> places, the largest height first
        const int warps = (n_expert + 32) / 32;
        int c = 0;
        for (int w = 0; w < warps; w++) c += first[w][lane];
        if (lane == 0) c = 0;
        int ge = c; // tiles of this height and the larger ones
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int a = __shfl_down_sync(0x0000ffffu, ge, o, 16);
            if (lane + o < 16) ge += a;
        }
        int at = ge - c;
        for (int w = 0; w < warps; w++) {
            const int m = first[w][lane];
            first[w][lane] = at;
            at += m;
        }
        if (lane == 0) *n_tiles = min(ge, max_tiles);
    }
    __syncthreads();
    const int r0 = cr - rows + (warp ? warp_sum[warp - 1] : 0);
    if (n == 1) { // (the whole list, whatever the height)
        const int t = first[warp][low] + at_low;
        if (t < max_tiles) tiles[t] = make_int4(e, 0, rows, r0);
        return;
    }
    for (int i = 0; i < n; i++) {
        const bool high = i < high_n;
        const int t = high ? first[warp][low + 1] + at_high + i : first[warp][low] + at_low + i - high_n;
        const int l0 = 16 * (i * low + min(i, high_n));
        if (t < max_tiles) tiles[t] = make_int4(e, l0, min(16 * (low + high), rows - l0), r0 + l0);
    }
}

// Routed rows -> the f16 B operand in TILE ORDER.  Row tile `slot` (nt routed rows of one expert)
// and k-stage ks (64 values) form one contiguous block of nt * 128 bytes that is the exact shared-memory image
// of a B stage: row rr at rr*128 B, its 16-byte chunk c at position c ^ (rr & 7) (the 128-byte
// swizzle of the tensor core's K-major layout), 8 values per chunk in the order [0 2 1 3 4 6 5 7]
// (the order in which the dequantiser emits a chunk of weights).  A B stage is then ONE bulk copy.
// (Tile::gather4 loads straight from token order take 62 cycles for four rows, 2960 for the 192 rows of a stage that is
// multiplied in 770.)
// pos[flat id] = slot*nt + rr lets later kernels (SwiGLU) write rows in the same order.
__device__ __forceinline__ size_t tiled_off(int slot, int k_stages, int ks, int rr, int c, int nt) {
    return (((size_t)slot * k_stages + ks) * nt + rr) * 128 + ((size_t)(c ^ (rr & 7)) << 4);
}

// A block takes GT_ROWS rows of one row tile, one warp per row: the work is even however the rows fall to the experts, and no
// row waits behind another of its warp (5120 rows of 3072 in 256 tiles: 32 rows a block 25.6 us, 8 rows 12.7).
constexpr int GT_ROWS = 8;
template <bool XF16>
__global__ void __launch_bounds__(256) gather_tiles_kernel(const void *__restrict__ xv, int x_per_row, int top_k, int k,
                                                           const int4 *__restrict__ tiles, const int32_t *__restrict__ n_tiles,
                                                           const int32_t *__restrict__ ids_map, int map_stride, int n_expert,
                                                           int routed_rows, int nt, uint8_t *__restrict__ xt,
                                                           int32_t *__restrict__ pos, int32_t *__restrict__ spos,
                                                           int32_t *__restrict__ sfid) {
    pdl_begin();
    const int slot = blockIdx.x;
    if (slot >= *n_tiles) return;
    const int4 T = tiles[slot];
    const int lane = threadIdx.x & 31, k_stages = k / MM_K, chunks = k / 8;
    const int end = min(T.z, (int)(blockIdx.y + 1) * GT_ROWS);
    for (int rr = blockIdx.y * GT_ROWS + (threadIdx.x >> 5); rr < end; rr += 8) {
        const bool shared = T.x == n_expert; // the shared expert's rows are the tokens in order, their ids follow the routed ones
        const int fid = shared ? routed_rows + T.y + rr : ids_map[(size_t)T.x * map_stride + T.y + rr];
        const size_t srow = (size_t)(shared ? T.y + rr : (x_per_row == 1 ? fid / top_k : fid)) * k;
        if (lane == 0) {
            if (pos) pos[fid] = slot * nt + rr;
            if (spos) spos[fid] = T.w + rr;
            if (sfid) sfid[T.w + rr] = fid;
        }
#pragma unroll 4
        for (int ci = lane; ci < chunks; ci += 32) {
            uint4 o;
            if (XF16) {
                // rows already in f16 (the expert-parallel wire format): only the order inside the chunk changes
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(static_cast<const __half *>(xv) + srow) + ci);
                o = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410),
                               __byte_perm(v.z, v.w, 0x7632));
            } else {
                const float *src = static_cast<const float *>(xv) + srow;
                const float4 a = __ldg(reinterpret_cast<const float4 *>(src) + 2 * ci);
                const float4 b = __ldg(reinterpret_cast<const float4 *>(src) + 2 * ci + 1);
                __align__(16) __half2 h[4] = {__floats2half2_rn(a.x, a.z), __floats2half2_rn(a.y, a.w),
                                              __floats2half2_rn(b.x, b.z), __floats2half2_rn(b.y, b.w)};
                o = *reinterpret_cast<const uint4 *>(h);
            }
            *reinterpret_cast<uint4 *>(xt + tiled_off(slot, k_stages, ci >> 3, rr, ci & 7, nt)) = o;
        }
    }
}

// The gate/up product takes its activation rows straight from token order: x once as f16 [tokens][k] (8-value chunks as
// [0 2 1 3 4 6 5 7]), and src[slot * nt + rr] = row of it that tile row (slot, rr) multiplies.  The kernel's loaders fetch the
// rows of every 64-k block with 16-byte asynchronous copies; a row of a token that ten experts share stays in L2 instead of
// being written out and read back ten times.  Blocks [0, convert_blocks) convert x, the others take a row tile each.
template <bool XF16>
__global__ void __launch_bounds__(256) stage_rows_kernel(const void *__restrict__ xv, int64_t x_chunks, int convert_blocks, int top_k,
                                                         const int4 *__restrict__ tiles, const int32_t *__restrict__ n_tiles,
                                                         const int32_t *__restrict__ ids_map, int map_stride, int n_expert,
                                                         int routed_rows, int nt, uint8_t *__restrict__ xh, int32_t *__restrict__ src,
                                                         int32_t *__restrict__ pos, int32_t *__restrict__ spos, int32_t *__restrict__ sfid) {
    pdl_begin();
    if ((int)blockIdx.x < convert_blocks) {
        const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
        if (i >= x_chunks) return;
        uint4 o;
        if (XF16) {
            // rows already in f16 (the expert-parallel wire format): only the order inside the chunk changes
            const uint4 v = __ldg(static_cast<const uint4 *>(xv) + i);
            o = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410),
                           __byte_perm(v.z, v.w, 0x7632));
        } else {
            const float4 a = __ldg(static_cast<const float4 *>(xv) + 2 * i), b = __ldg(static_cast<const float4 *>(xv) + 2 * i + 1);
            __align__(16) __half2 h[4] = {__floats2half2_rn(a.x, a.z), __floats2half2_rn(a.y, a.w), __floats2half2_rn(b.x, b.z),
                                          __floats2half2_rn(b.y, b.w)};
            o = *reinterpret_cast<const uint4 *>(h);
        }
        reinterpret_cast<uint4 *>(xh)[i] = o;
        return;
    }
    const int slot = blockIdx.x - convert_blocks, rr = threadIdx.x;
    if (slot >= *n_tiles) return;
    const int4 T = tiles[slot];
    if (rr >= T.z) return;
    const bool shared = T.x == n_expert; // the shared expert's rows are the tokens in order, their ids follow the routed ones
    const int fid = shared ? routed_rows + T.y + rr : ids_map[(size_t)T.x * map_stride + T.y + rr];
    src[slot * nt + rr] = shared ? T.y + rr : fid / top_k;
    pos[fid] = slot * nt + rr;
    if (spos) spos[fid] = T.w + rr;
    if (sfid) sfid[T.w + rr] = fid;
}

// ---- the grouped GEMM kernel -------------------------------------------------------------
// One kernel, three uses: NPROJ = 2 multiplies a block of routed rows by 128 gate rows AND the matching 128 up
// rows (every activation stage is loaded once for both, SwiGLU in the epilogue); NPROJ = 1 is a single
// projection (the down projection, and the op-level `mul_mm_id` of either format).
//
// Sixteen dequantising warps in two groups of eight take the pipeline stages in turn.  A stage is 64 weights for
// each of a group's 256 threads, 2 projections x 128 rows x 64 k or 128 rows x 128 k, and with tiles of up to 128 rows
// (WIDE) twice that.  The f16 values go straight
// into TENSOR MEMORY (tcgen05.st: lane = weight row) and the tensor core takes its A operand from there (TS form),
// so the dequantised tile never passes through shared memory.  A thread converts its next stage's weights BEFORE it
// waits for the stage to be free, so the wait covers only the store.
// A thin tile is bound by instructions, on the converting warps' schedulers as a whole (70 % of the issue slots, of the integer pipe
// 64) and one by one in the warp that issues the multiplies (450 to 560 cycles a stage where its multiplies take 100): hence the wide stages, which halve
// what is done once a stage, tc_mma_block's assembly, and subnormal operands in the conversion.  A block's forward with its shared
// expert, 128 / 512 / 1024 / 2048 tokens on 256 experts of 1024, cold L2: 402 / 489 / 591 / 840 us with stages of 64 weights and the
// plain conversion, 382 / 470 / 579 / 813 with wide stages and lean issue, 365 / 452 / 554 / 800 with the subnormal conversion
// too; 318 without conversions at 128 tokens, 240 the weights at the copy rate.  Four groups of four warps (396 / 483 / 589), the next
// stage's words loaded ahead (411 / 517 / 623: the operand slots are held for longer) and other ways of waiting (none shorter) were tried.
//
// Two CTAs on neighbouring SMs share a tile (CG = 2, cta_group::2; with CG = 1 a CTA has a tile of 128 weight rows for itself): each
// converts 128 of its 256 weight rows and keeps their accumulators, and each loads half of the tile's activation rows, which the tensor cores of both read.  One SM alone loads 24 KB of
// activations for 768 cycles of multiplies in gate/up, 48 KB in down, and with the weights that is more than the L2 cache hands
// out: down of 8192 tokens took the same 990 thousand cycles without its conversions or with 16-column multiplies.  The first CTA's
// warp 0 issues for both; whatever it waits for is signalled at its barriers by both CTAs, and its commits arrive in both.  (What is
// handed over lies in tensor memory, behind tcgen05 fences, or in a CTA's own shared memory, behind a proxy fence or a bulk copy's
// completion, so the arrivals are of the default scope: with release and acquire at cluster scope a signal took over a thousand
// cycles.)
//
// The multiplies are issued by an elected lane inside a loop that the whole warp runs: the operand addresses then
// stay in uniform registers.  Issued from a lane == 0 branch a tcgen05.mma costs 46 cycles of issue whatever its
// width; this way a 16-column one takes 10 and an N-column one N/2, the tensor core's own rate.
//
// Tensor-memory columns: [0, NT) and [NT, 2 NT): the gate and up accumulators, or the two accumulator
// buffers of a single projection (its epilogue runs beside the next tile's multiplies); the rest holds the operand
// stages: two of 64 columns beside 192-row tiles, of 128 columns two beside 128-row and three beside 64-row tiles.
//   warp 0    MMA issuer (second CTA, single projection: relay)    warp 2 loader of the quantized columns    warps 8-23 dequant
//   single projection: warp 1 B loader (bulk copies of the tile-ordered operand), warps 4-7 epilogue
//   two projections: warps 4-7 B loaders (rows in token order), the epilogue falls to the dequantising warps
constexpr int GM_DQ_WARPS = 16, GM_DQ0 = 8; // number of dequantising warps, the first of them
constexpr int GM_THREADS = (GM_DQ_WARPS + 8) * 32;
// A 210-byte block inside its 224-byte aligned window; neighbouring lines lie in different banks (60 words).
constexpr int GM_Q6_PITCH = 240;
constexpr int GM_Q6_COPY = 224;
// 2^lg rows of n_blk 210-byte blocks are the least that a multiple of 16 bytes holds: the lines of the tile loads.  As few as
// that, because 2^lg - 1 neighbours of a row lie 128 / 2^lg lines away, in its own banks but for the block's offset in its granule.
__host__ __device__ __forceinline__ int gm_q6_lg(int n_blk) { return n_blk & 1 ? 3 : (n_blk & 2 ? 2 : (n_blk & 4 ? 1 : 0)); }
// the line of row r of a tile
__device__ __forceinline__ int gm_q6_line(int r, int lg) { return ((r & ((1 << lg) - 1)) << (7 - lg)) + (r >> lg); }
constexpr int GM_EPI_BYTES = 1024; // one epilogue warp's staging: 8 tile columns (output rows) x 32 weight rows, f32
constexpr int GM_BOX_ROWS = 16;    // single projection: tile stores of 16 output rows x 32 weight rows, two in flight per warp

template <int DT, int NPROJ, int NT, int CG>
struct GmCfg {
    // one 256-wide column of quantized blocks of all the tile's weight rows
    static constexpr int RAW_SLOT = NPROJ * MM_M * (DT == LMOE_Q4_K ? Q4K_BYTES : GM_Q6_PITCH);
    static constexpr int RAW_SLOTS = DT == LMOE_Q4_K && NPROJ == 1 ? 4 : 3;
    static constexpr int EPI_BYTES = NPROJ == 2 ? GM_EPI_BYTES : 2 * GM_BOX_ROWS * 128;
    static constexpr int B_ROWS = NT / CG;
    static constexpr int B_BLK = B_ROWS * MM_K * 2;     // a CTA's half of a 64-k block of the B operand
    // blocks of a full tile in a ring slot (two in the slots of gate/up's 128-row tiles, three runs in turn: 64 experts of 1536, hidden 4096,
    // 176 / 280 / 400 tokens 285.5 / 295.0 / 310.3 -> 283.6 / 291.8 / 306.1 us, 256 experts of 1024 0.5 to 1.5 % where two runs differ by 1)
    static constexpr int B_FULL = (NPROJ == 2 || CG == 1 ? 1 : 2) * (NT == 64 || (NPROJ == 2 && NT == 128) ? 2 : 1);
    static constexpr int B_SLOT = B_FULL * B_BLK;
    static constexpr int NB = 96 * 1024 / B_SLOT < 8 ? 96 * 1024 / B_SLOT : 8;
    static constexpr bool WIDE = NT <= 128;             // operand stages of 128 weights a thread, else 64
    static constexpr int A_COLS = WIDE ? 128 : 64, NA = (512 - 2 * NT) / A_COLS, A_COL0 = 2 * NT;
    static constexpr int A_BLKS = (WIDE ? 2 : 1) * (NPROJ == 2 ? 1 : 2); // 64-k blocks of an operand stage
    static constexpr int RAW_READERS = WIDE && NPROJ == 1 ? GM_DQ_WARPS / 2 : GM_DQ_WARPS;
    static constexpr int EPI_WARPS = NPROJ == 2 ? GM_DQ_WARPS : 4;
    static constexpr int B_ARRIVALS = NPROJ == 2 ? 4 * CG : 1; // per ring slot (the first CTA's of a single projection: one more, see the relay)
    static constexpr int O_RAW = NB * B_SLOT, O_EPI = O_RAW + RAW_SLOTS * RAW_SLOT, O_BAR = O_EPI + EPI_WARPS * EPI_BYTES;
    static constexpr int SMEM = O_BAR + 512 + 1024; // barriers, slack to align the base to 1024 bytes
    static_assert(A_COL0 + A_COLS * NA <= 512 && NA >= 2, "tensor memory");
    static_assert(SMEM <= 227 * 1024, "shared memory");
};

struct GmParams {
    // Q4_K: 2-D byte views [n_expert * n_out rows][row_bytes], box = 144 bytes x 128 rows.
    // Q6_K (n_out a multiple of 2^lg, see gm_q6_lg): 2^lg rows as one line, box = 240 bytes x 128 / 2^lg lines
    // [0, 1]: the experts' stacks (gate / up, or one projection), [2, 3]: the shared expert's
    CUtensorMap map[4];
    CUtensorMap map_out;     // NPROJ = 1, sorted rows: `out` as [rows][n_out] f32, box = 32 values x 16 rows
    int lines, lg;           // Q6_K: the views exist; lg
    const uint8_t *w[2];     // Q6_K without them: stack blocks, shared expert's blocks
    int n_expert, m_tiles;   // list number of the shared expert; blocks of CG x 128 weight rows
    int64_t expert_bytes;
    int n_out, k;
    const uint8_t *xt;       // NPROJ = 1: f16 activations in tile order (see gather_tiles_kernel); 2: in token order
    const int32_t *src;      // NPROJ = 2: row of xt of every tile row (see stage_rows_kernel)
    const int32_t *ids_map;  // [n_expert, map_stride] flat ids
    int map_stride;
    const int4 *tiles;       // row tiles, see row_tiles_kernel
    const int32_t *n_tiles;
    const float *row_scale;  // per flat id, or NULL (NPROJ = 1, rows by flat id)
    float *out;              // rows of n_out values
    int sorted;              // rows of `out` in expert-sorted order, unscaled, instead of by flat id
    int vec;                 // n_out and `out` allow 16-byte stores
    uint32_t *flag;
};

// 64 weights (sub-block pair j) of one Q4_K row -> 32 words, in the order the activation rows are stored
// (8-value chunks as [0 2 1 3 4 6 5 7]): word 4c + i = chunk c, pair i.
// The scale d * sc and the offset -dmin * m are products of an f16 and a six-bit integer, rounded once to f16.
// `small` (|d| < 2^-10, so that every scale is below 2^-4): a nibble in bits 4 to 7 of a half is the subnormal q * 2^-20, and the fma
// takes it as it is with the scale times 2^20: the same product, so the same value, without the subtraction that makes a plain q.
constexpr uint32_t Q4K_SMALL_D = 0x1400; // f16 bits of 2^-10
__device__ __forceinline__ void dequant_q4k_regs(const uint4 hdr, const uint4 qa, const uint4 qb, int j, bool small, uint32_t (&o)[32]) {
    uint32_t sc[2], mn[2];
    q4k_unpack_scales(hdr.y, hdr.z, hdr.w, sc[0], sc[1], mn[0], mn[1]);
    // bytes 2 (j & 1), 2 (j & 1) + 1 of word j >> 1 -> 1024 + value, as an f16 pair
    const uint32_t sel = (j & 1) ? 0x4342u : 0x4140u;
    const uint32_t d2 = prmt(hdr.x, 0u, 0x1010u);
    uint32_t s2 = h2_sub_mul(prmt((j & 2) ? sc[1] : sc[0], 0x64646464u, sel), 0x64006400u, small ? h2_mul(d2, 0x64006400u) : d2);
    const uint32_t m2 = h2_sub_mul(prmt((j & 2) ? mn[1] : mn[0], 0x64646464u, sel), 0x64006400u, prmt(hdr.x ^ 0x80000000u, 0u, 0x3232u));
    const uint32_t m_lo = prmt(m2, 0u, 0x1010u), m_hi = prmt(m2, 0u, 0x3232u);
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
    if (small) {
        s2 = h2_mul(s2, 0x64006400u);
        const uint32_t s_lo = prmt(s2, 0u, 0x1010u), s_hi = prmt(s2, 0u, 0x3232u);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const uint32_t v = w[c];
            // low nibbles (sub-block 2j): chunks 0-3; high nibbles (sub-block 2j+1): chunks 4-7
            o[2 * c] = h2_fma((v << 4) & 0x00F000F0u, s_lo, m_lo);
            o[2 * c + 1] = h2_fma((v >> 4) & 0x00F000F0u, s_lo, m_lo);
            o[16 + 2 * c] = h2_fma(v & 0x00F000F0u, s_hi, m_hi);
            o[16 + 2 * c + 1] = h2_fma((v >> 8) & 0x00F000F0u, s_hi, m_hi);
        }
        return;
    }
    const uint32_t s_lo = prmt(s2, 0u, 0x1010u), s_hi = prmt(s2, 0u, 0x3232u);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const uint32_t v = w[c], v8 = v >> 8;
        // the same nibbles as 1024 + q and, in place, 64 + q
        o[2 * c] = h2_sub_fma(and_or(v, 0x000F000Fu, 0x64006400u), 0x64006400u, s_lo, m_lo);
        o[2 * c + 1] = h2_sub_fma(and_or(v8, 0x000F000Fu, 0x64006400u), 0x64006400u, s_lo, m_lo);
        o[16 + 2 * c] = h2_sub_fma(and_or(v, 0x00F000F0u, 0x54005400u), 0x54005400u, s_hi, m_hi);
        o[16 + 2 * c + 1] = h2_sub_fma(and_or(v8, 0x00F000F0u, 0x54005400u), 0x54005400u, s_hi, m_hi);
    }
}

// 16 bytes at byte offset `o` (even) from a 4-byte aligned base, as four words
__device__ __forceinline__ void read16_a2(const uint8_t *base4, int o, uint32_t (&out)[4]) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(base4) + (o >> 2);
    const uint32_t sh = (uint32_t)(o & 3) * 8u;
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
    out[0] = __funnelshift_r(w0, w1, sh);
    out[1] = __funnelshift_r(w1, w2, sh);
    out[2] = __funnelshift_r(w2, w3, sh);
    out[3] = __funnelshift_r(w3, w4, sh);
}

// The fields of half n, l range lh (16 wide) of the Q6_K block that starts `sh` bytes (even) after the 4-byte aligned
// address base4: 16 bytes of ql for groups {0, 2} and {1, 3}, 16 bytes of qh, the half's eight scales, d (both halves of the word).
struct Q6Fields {
    uint32_t qa[4], qb[4], qh[4], s0, s1, d2;
};
__device__ __forceinline__ void q6k_fields(const uint8_t *base4, int sh, int n, int lh, Q6Fields &F) {
    read16_a2(base4, sh + 64 * n + 16 * lh, F.qa);
    read16_a2(base4, sh + 64 * n + 32 + 16 * lh, F.qb);
    read16_a2(base4, sh + 128 + 32 * n + 16 * lh, F.qh);
    const int p = sh + 192 + 8 * n;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(base4) + (p >> 2);
    const uint32_t s = (uint32_t)(p & 3) * 8u;
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
    F.s0 = __funnelshift_r(w0, w1, s);
    F.s1 = __funnelshift_r(w1, w2, s);
    F.d2 = prmt(reinterpret_cast<const uint32_t *>(base4)[(sh + 208) >> 2], 0u, (sh & 2) ? 0x3232u : 0x1010u);
}
// The same where a row's blocks are a multiple of 8 bytes (rows of 4 i blocks): the offset of block b in its granule is 2 b bytes
// modulo 8 for every row of the tile, so the words come in pairs and a branch that all lanes take alike picks them.  The tile's
// lines (gm_q6_line) then put sixteen lanes' pairs into different banks at k = 1024 and 3072 (two lanes' into the same at 2048
// and 4096): 24 shared-memory passes a warp and block where single words of lines of eight rows took 76 (at 2048: 152), beside
// the tensor core's own reads the bound of the down product.
__device__ __forceinline__ void q6k_fields_paired(const uint8_t *base8, int sh, int b, int n, int lh, Q6Fields &F) {
    const uint2 *w = reinterpret_cast<const uint2 *>(base8) + ((sh & 8) >> 3) + 8 * n + 2 * lh;
    const uint2 *ws = reinterpret_cast<const uint2 *>(base8) + ((sh & 8) >> 3) + 24 + n;
    const uint2 a0 = w[0], a1 = w[1], a2 = w[2], b0 = w[4], b1 = w[5], b2 = w[6];
    const uint2 *wh = w + 16 - 4 * n;
    const uint2 h0 = wh[0], h1 = wh[1], h2 = wh[2], s0 = ws[0], s1 = ws[1], s2 = ws[n ? 1 : 2];
    const uint32_t s = (uint32_t)(b & 1) * 16u, dsel = (b & 1) ? 0x3232u : 0x1010u;
    if (b & 2) {
        F.qa[0] = __funnelshift_r(a0.y, a1.x, s); F.qa[1] = __funnelshift_r(a1.x, a1.y, s);
        F.qa[2] = __funnelshift_r(a1.y, a2.x, s); F.qa[3] = __funnelshift_r(a2.x, a2.y, s);
        F.qb[0] = __funnelshift_r(b0.y, b1.x, s); F.qb[1] = __funnelshift_r(b1.x, b1.y, s);
        F.qb[2] = __funnelshift_r(b1.y, b2.x, s); F.qb[3] = __funnelshift_r(b2.x, b2.y, s);
        F.qh[0] = __funnelshift_r(h0.y, h1.x, s); F.qh[1] = __funnelshift_r(h1.x, h1.y, s);
        F.qh[2] = __funnelshift_r(h1.y, h2.x, s); F.qh[3] = __funnelshift_r(h2.x, h2.y, s);
        F.s0 = __funnelshift_r(s0.y, s1.x, s); F.s1 = __funnelshift_r(s1.x, s1.y, s);
        F.d2 = prmt(s2.y, 0u, dsel);
    } else {
        F.qa[0] = __funnelshift_r(a0.x, a0.y, s); F.qa[1] = __funnelshift_r(a0.y, a1.x, s);
        F.qa[2] = __funnelshift_r(a1.x, a1.y, s); F.qa[3] = __funnelshift_r(a1.y, a2.x, s);
        F.qb[0] = __funnelshift_r(b0.x, b0.y, s); F.qb[1] = __funnelshift_r(b0.y, b1.x, s);
        F.qb[2] = __funnelshift_r(b1.x, b1.y, s); F.qb[3] = __funnelshift_r(b1.y, b2.x, s);
        F.qh[0] = __funnelshift_r(h0.x, h0.y, s); F.qh[1] = __funnelshift_r(h0.y, h1.x, s);
        F.qh[2] = __funnelshift_r(h1.x, h1.y, s); F.qh[3] = __funnelshift_r(h1.y, h2.x, s);
        F.s0 = __funnelshift_r(s0.x, s0.y, s); F.s1 = __funnelshift_r(s0.y, s1.x, s);
        F.d2 = prmt(s2.x, 0u, dsel);
    }
}
// 16 weights of each of the half's four 32-wide groups -> o[8 g .. 8 g + 7] = group g's values 16 lh .. 16 lh + 15,
// 8-value chunks as [0 2 1 3 4 6 5 7].  Four six-bit values are put together per word (low nibble | two high bits << 4),
// then spread two at a time into f16 pairs 1024 + q by one byte permute; q - 32 is exact and the scale rounds once.
// `small` (|d| < 2^-13, so that every scale is below 2^-6): the values stand two bits higher in their bytes, as the subnormals q * 2^-22,
// and one fma with the scale times 2^22 and -32 scales gives the same value.
constexpr uint32_t Q6K_SMALL_D = 0x0800; // f16 bits of 2^-13
__device__ __forceinline__ void dequant_q6k_regs(const Q6Fields &F, int lh, bool small, uint32_t (&o)[32]) {
    // the four groups' scales are bytes lh, 2 + lh of s0 and of s1, signed: (s ^ 0x80) + 1024 - 1152
    const uint32_t selp = lh ? 0x4341u : 0x4240u;
    const uint32_t d2 = small ? h2_mul(F.d2, 0x78007800u) : F.d2; // * 2^15
    const uint32_t sc01 = h2_sub_mul(prmt(F.s0 ^ 0x80808080u, 0x64646464u, selp), 0x64806480u, d2);
    const uint32_t sc23 = h2_sub_mul(prmt(F.s1 ^ 0x80808080u, 0x64646464u, selp), 0x64806480u, d2);
    if (small) {
        const uint32_t b01 = h2_mul(sc01, 0x94009400u), b23 = h2_mul(sc23, 0x94009400u); // * -2^-10: -32 scales
        const uint32_t m01 = h2_mul(sc01, 0x58005800u), m23 = h2_mul(sc23, 0x58005800u); // * 2^7
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const uint32_t sel = (g & 1) ? 0x3232u : 0x1010u;
            const uint32_t sc = prmt(g < 2 ? m01 : m23, 0u, sel), off = prmt(g < 2 ? b01 : b23, 0u, sel);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t q = (g & 1) ? F.qb[j] : F.qa[j], ql = g < 2 ? q << 2 : q >> 2;
                const uint32_t h = g == 0 ? F.qh[j] << 6 : (g == 1 ? F.qh[j] << 4 : (g == 2 ? F.qh[j] << 2 : F.qh[j]));
                const uint32_t q6 = and_or(ql, 0x3C3C3C3Cu, h & 0xC0C0C0C0u);
                o[8 * g + 2 * j] = h2_fma(prmt(q6, 0u, 0x4240u), sc, off);
                o[8 * g + 2 * j + 1] = h2_fma(prmt(q6, 0u, 0x4341u), sc, off);
            }
        }
        return;
    }
    const uint32_t off = 0x64206420u; // 1024 + 32
#pragma unroll
    for (int g = 0; g < 4; g++) {
        // groups 0, 1: low nibbles of qa, qb; groups 2, 3: their high nibbles
        const uint32_t sc = prmt(g < 2 ? sc01 : sc23, 0u, (g & 1) ? 0x3232u : 0x1010u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t q = (g & 1) ? F.qb[j] : F.qa[j], ql = g < 2 ? q : q >> 4;
            const uint32_t h = g == 0 ? F.qh[j] << 4 : (g == 1 ? F.qh[j] << 2 : (g == 2 ? F.qh[j] : F.qh[j] >> 2));
            const uint32_t q6 = and_or(ql, 0x0F0F0F0Fu, h & 0x30303030u);
            o[8 * g + 2 * j] = h2_sub_mul(prmt(q6, 0x64646464u, 0x4240u), off, sc);
            o[8 * g + 2 * j + 1] = h2_sub_mul(prmt(q6, 0x64646464u, 0x4341u), off, sc);
        }
    }
}

// One entry of the tile table.  Every role reads the entry of its next tile while it works on the current one: a table
// read costs most of a microsecond, a fifth of a thin tile's whole time.
struct GmTile {
    int e, sh; // expert; 1 for the shared expert (then e is 0)
    int l0, nv, m0, slot, srow;
};
template <int CG>
__device__ __forceinline__ GmTile gm_tile(const GmParams &P, int tile, int n_tiles, int rank) {
    GmTile T = {0, 0, 0, 0, 0, 0, 0};
    if (tile < n_tiles) {
        const int slot = tile / P.m_tiles;
        const int4 a = __ldg(P.tiles + slot);
        const int sh = a.x == P.n_expert;
        T = {sh ? 0 : a.x, sh, a.y, a.z, (tile - slot * P.m_tiles) * (CG * MM_M) + rank * MM_M, slot, a.w};
    }
    return T;
}
// 64-k blocks of the B operand that share one ring slot: a thin tile's blocks do not fill it, and a deeper ring is what
// hides the copies' latency there.
template <int FULL, int NT>
__device__ __forceinline__ int gm_b_group(int nv) {
    return nv > NT / 2 ? FULL : (FULL == 1 && nv > NT / 4 ? 2 : 4);
}

// rows of a tile that each CTA of a pair holds of the B operand (of the padded tile: a multiple of 8)
template <int CG>
__device__ __forceinline__ int gm_half(int nv) { return ((nv + 15) & ~15) / CG; }
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Epilogue of the 16-column chunks c0, c0 + cs, ... of a tile for the 32 weight rows of tensor-memory quadrant q: one
// output row per tile column.  NPROJ = 2: out = silu(gate) * up.  A lane holds one weight row, so eight columns at a
// time pass through the warp's staging buffer and leave as 16-byte stores, 128 contiguous bytes per output row
// (4-byte stores straight from the registers kept the down projection waiting for its epilogue: 390 us against 255
// without one at 4096 tokens).
template <int NPROJ, int NT>
__device__ __forceinline__ void gm_epilogue(const GmParams &P, const GmTile &T, uint32_t acc0, float *stage, int q, int lane, int c0, int cs) {
    const int m = T.m0 + 32 * q, nv = T.nv;
    const uint32_t t0 = acc0 + ((uint32_t)(32 * q) << 16);
    const size_t ld = (size_t)P.n_out;
    const int32_t *list = P.ids_map + (size_t)T.e * P.map_stride + T.l0;
    const int sub = lane >> 3, seg = 4 * (lane & 7); // this lane's part of a store: row sub (+ 4), values seg .. seg + 3
    int c = c0;
    if (NPROJ == 1 && P.sorted && P.vec && m + 32 <= P.n_out) {
        // whole chunks of 16 rows leave through the tensor-memory-access unit: one instruction per kilobyte pair instead of
        // a load, an address and a store for every 512 bytes (the four epilogue warps had more to issue than a tile's
        // multiplies take)
        const bool el = elect_one();
        for (int i = 0; 16 * (c + 1) <= nv; c += cs, i ^= 1) {
            uint32_t v[16];
            tc_ld16(t0 + 16 * c, v);
            float *buf = stage + i * (GM_BOX_ROWS * 32);
            if (el) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); // the store before last has left this buffer
            __syncwarp();
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; j++) buf[32 * j + lane] = __uint_as_float(v[j]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (el) {
                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&P.map_out), "r"(m),
                             "r"(T.srow + 16 * c), "r"(s32(buf)) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (el) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
    }
    for (; 16 * c < nv; c += cs) {
        const int cb = 16 * c;
        int fid[4];
        float sc[4];
        if (!P.sorted) {
#pragma unroll
            for (int i = 0; i < 4; i++) fid[i] = cb + sub + 4 * i < nv ? list[cb + sub + 4 * i] : 0;
        }
        uint32_t v[16], u[16];
        tc_ld16(t0 + cb, v);
        if (NPROJ == 2) tc_ld16(t0 + NT + cb, u);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; i++) sc[i] = (NPROJ == 1 && !P.sorted && P.row_scale) ? P.row_scale[fid[i]] : 1.0f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float gv = __uint_as_float(v[8 * h + j]);
                stage[32 * j + lane] = NPROJ == 2 ? __fdividef(gv, 1.0f + __expf(-gv)) * __uint_as_float(u[8 * h + j]) : gv;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int row = cb + 8 * h + 4 * i + sub;
                float4 o = *reinterpret_cast<const float4 *>(stage + 32 * (4 * i + sub) + seg);
                const size_t orow = P.sorted ? (size_t)(T.srow + row) : (size_t)fid[2 * h + i];
                float *dst = P.out + orow * ld + m + seg;
                if (NPROJ == 1) { o.x *= sc[2 * h + i]; o.y *= sc[2 * h + i]; o.z *= sc[2 * h + i]; o.w *= sc[2 * h + i]; }
                if (row < nv) {
                    if (P.vec) {
                        if (m + seg < P.n_out) *reinterpret_cast<float4 *>(dst) = o;
                    } else {
                        if (m + seg < P.n_out) dst[0] = o.x;
                        if (m + seg + 1 < P.n_out) dst[1] = o.y;
                        if (m + seg + 2 < P.n_out) dst[2] = o.z;
                        if (m + seg + 3 < P.n_out) dst[3] = o.w;
                    }
                }
            }
        }
    }
}

template <int DT, int NPROJ, int NT, int CG>
__global__ void __launch_bounds__(GM_THREADS, 1) grouped_mm_kernel(const __grid_constant__ GmParams P) {
    using C = GmCfg<DT, NPROJ, NT, CG>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *b_st = smem, *raw = smem + C::O_RAW;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::O_BAR);
    // a_full[s]: the eight warps of the stage's group, of both CTAs; a_empty[s]: one commit; b_full[i]: the copies' bytes, or both CTAs'
    // loaders; b_empty[i]: one commit;
    // raw_full[i]: the copies' bytes; raw_empty[i]: the dequantising warps that read it, all sixteen or the eight of a
    // group (RAW_READERS); acc_*: per accumulator buffer
    uint64_t *a_full = bars, *a_empty = bars + 4, *b_full = bars + 8, *b_empty = bars + 16, *raw_full = bars + 24,
             *raw_empty = bars + 28, *acc_full = bars + 32, *acc_empty = bars + 34;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 36);
    static_assert(C::NB <= 8 && C::RAW_SLOTS <= 4 && C::NA <= 4, "barrier table");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = CG == 2 ? blockIdx.x & 1 : 0, tile0 = blockIdx.x / CG, tile_step = gridDim.x / CG; // place in the pair; the pair's tiles
    const int n_blk = P.k / QK_K, k_blocks = P.k / MM_K;
    const int row_bytes = n_blk * (DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES);

    if (tid == 0) {
        for (int s = 0; s < C::NA; s++) {
            mb_init(&a_full[s], GM_DQ_WARPS / 2 * CG);
            mb_init(&a_empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mb_init(&acc_full[s], 1);
            mb_init(&acc_empty[s], CG * C::EPI_WARPS);
        }
        for (int i = 0; i < C::NB; i++) {
            mb_init(&b_full[i], C::B_ARRIVALS + (NPROJ == 1 && CG == 2 && rank == 0 ? 1 : 0));
            mb_init(&b_empty[i], 1);
        }
        for (int i = 0; i < C::RAW_SLOTS; i++) {
            mb_init(&raw_full[i], 1);
            mb_init(&raw_empty[i], C::RAW_READERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        if (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) pair_sync(); // the other CTA's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory"); // what earlier kernels wrote is read from here on
    const int n_tiles = *P.n_tiles * P.m_tiles;
    bool ok = true; // false once a wait of this warp has run out
    // A loader leaves when its copies have landed, also where their readers have given up: slot i < next was filled in the present turn of
    // the ring (its parity), the others in the turn before (a barrier never used counts as complete).
    auto landed = [&](uint64_t *full, int n, uint32_t next, uint32_t parity) {
        bool here = true;
        for (int i = 0; i < n && here; i++) here = mb_wait(&full[i], (uint32_t)i < next ? parity : parity ^ 1);
        ok &= here;
    };

    if (warp >= GM_DQ0) {
        // ---------------- dequant: thread = (part, weight row), group = stage parity ----------------
        // part: the projection (NPROJ = 2), the 64-wide k half of a stage (Q4_K) or the 16-wide l range (Q6_K)
        const int grp = (warp - GM_DQ0) >> 3, part = (warp >> 2) & 1, q = warp & 3, r = 32 * q + lane;
        const uint32_t ta = tmem_base + ((uint32_t)(32 * q) << 16) + C::A_COL0;
        float *stage = reinterpret_cast<float *>(smem + C::O_EPI + (NPROJ == 2 ? (warp - GM_DQ0) * C::EPI_BYTES : 0));
        uint32_t slot = C::WIDE && NPROJ == 1 ? grp : 0, rph = 0, it = 0; // raw ring slot and its phase, tiles
        uint32_t as = grp, aph = 0;                                      // operand slot of the group's next stage: every second one
        auto slot_free = [&]() {
            ok &= mb_wait(&a_empty[as], aph ^ 1);
            tc_fence_after();
        };
        auto stored = [&]() {
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive_first<CG>(&a_full[as]);
            if ((as += 2) >= C::NA) { as -= C::NA; aph ^= 1; }
        };
        auto read = [&]() { // this warp is done with the ring slot
            __syncwarp();
            if (lane == 0) mb_arrive(&raw_empty[slot]);
            if ((slot += C::WIDE && NPROJ == 1 ? 2 : 1) >= C::RAW_SLOTS) { slot -= C::RAW_SLOTS; rph ^= 1; }
        };
        int sh = 0; // Q6_K: offset of the block inside its 16-byte granule
        const uint32_t line = DT == LMOE_Q6_K ? (uint32_t)gm_q6_line(r, P.lg) * GM_Q6_PITCH : 0u;
        auto q6_fields = [&](int b, int n, Q6Fields &F) {
            const uint8_t *rs = raw + (size_t)slot * C::RAW_SLOT + line;
            if (P.lg <= 1) q6k_fields_paired(rs, sh, b, n, part, F);
            else q6k_fields(rs, sh & 15, n, part, F);
        };
        const uint32_t blk0 = (uint32_t)((NPROJ == 2 ? part * MM_M : 0) + r) * Q4K_BYTES;
        uint4 hdr, qw[C::WIDE ? 4 : 2];
        Q6Fields F[C::WIDE ? 2 : 1];
        // sub-block pair of the thread's first 64 weights of a column; a wide stage takes the next pair too
        const int j0 = C::WIDE ? 2 * (NPROJ == 2 ? grp : part) : (NPROJ == 2 ? grp : 2 * grp + part);
        // the thread's part of a stage, out of shared memory: sub-block pair j (and the next), or half n (both)
        auto fetch = [&](int j, int b) {
            if (DT == LMOE_Q4_K) {
                const uint4 *blk = reinterpret_cast<const uint4 *>(raw + (size_t)slot * C::RAW_SLOT + blk0);
                hdr = blk[0];
#pragma unroll
                for (int i = 0; i < (C::WIDE ? 4 : 2); i++) qw[i] = blk[1 + 2 * j + i];
            } else {
#pragma unroll
                for (int n = 0; n < (C::WIDE ? 2 : 1); n++) q6_fields(b, C::WIDE ? n : grp, F[n]);
            }
        };
        // 64 of its weights (half i of a wide stage) into the operand slot
        auto put = [&](const uint32_t (&o)[32], int i) {
            const uint32_t a = ta + (uint32_t)C::A_COLS * as;
            if (DT == LMOE_Q4_K) {
                tc_st32(a + (C::WIDE && NPROJ == 1 ? 64u * part + 32u * i : 64u * i + 32u * part), o);
            } else {
#pragma unroll
                for (int g = 0; g < 4; g++) tc_st8(a + 64u * i + 16u * g + 8u * part, o + 8 * g);
            }
        };
        bool small = false; // all the warp's rows have small scales in this column
        auto convert = [&](int j, int i, uint32_t (&o)[32]) {
            if (DT == LMOE_Q4_K) dequant_q4k_regs(hdr, qw[2 * i], qw[2 * i + 1], j + i, small, o);
            else dequant_q6k_regs(F[i], part, small, o);
        };
        auto stage_in = [&](int j) {
            small = __all_sync(0xffffffffu, DT == LMOE_Q4_K ? (hdr.x & 0x7FFFu) < Q4K_SMALL_D : (F[0].d2 & 0x7FFFu) < Q6K_SMALL_D);
            uint32_t o[32];
            convert(j, 0, o);
            slot_free();
            put(o, 0);
            if (C::WIDE) {
                uint32_t p[32];
                convert(j, C::WIDE ? 1 : 0, p);
                put(p, 1);
            }
        };
        // two projections: stage i of the group's one (wide) or two of a column
        auto part_of_column = [&](int i) {
            if (i == 0) ok &= mb_wait(&raw_full[slot], rph);
            fetch(j0 + 2 * i, 0);
            if (C::WIDE || i == 1) read();
            stage_in(j0 + 2 * i);
            stored();
        };
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        if (NPROJ == 2 && tile0 < n_tiles) part_of_column(0);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step, it++) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            // (rows past the last one convert whatever the slot holds: their accumulator rows are never read)
            if (NPROJ == 1) {
                // a wide stage is a whole column, and the groups take the columns in turn; else each takes its half of every column
                const int b0 = C::WIDE ? (grp ^ ((int)it * n_blk)) & 1 : 0, bs = C::WIDE ? 2 : 1;
                if (DT == LMOE_Q6_K) sh = (int)(((int64_t)T.e * P.expert_bytes + (int64_t)(T.m0 + r) * row_bytes) & 15) + b0 * Q6K_BYTES;
                auto load = [&](int b) {
                    ok &= mb_wait(&raw_full[slot], rph);
                    fetch(j0, b);
                    sh += bs * Q6K_BYTES;
                    read();
                };
                if (b0 < n_blk) load(b0);
                for (int b = b0; b < n_blk && ok; b += bs) {
                    stage_in(j0);
                    if (b + bs < n_blk) load(b + bs); // the next column's words arrive while the store completes
                    stored();
                }
            } else {
                // the rest of the tile's stages, then the first one of the next tile: it is there when
                // that tile's multiplies may begin (96 / 512 / 4096 / 16384 tokens 391 / 526 / 1343 / 4487 us without, 387 / 521 /
                // 1329 / 4447 so)
                for (int b = 0; b < n_blk && ok; b++) {
                    if (!C::WIDE) part_of_column(1);
                    if (b + 1 < n_blk || tile + tile_step < n_tiles) part_of_column(0);
                }
            }
            if (NPROJ == 2) {
                // this warp's share of the tile's epilogue: there is one accumulator set, so nothing is multiplied meanwhile
                const int c0 = (warp - GM_DQ0) >> 2;
                // (short rows: a group could run a whole tile ahead, so every warp waits here)
                if ((16 * c0 < T.nv || k_blocks <= 8) && ok) {
                    ok &= mb_wait(&acc_full[0], it & 1);
                    tc_fence_after();
                    gm_epilogue<NPROJ, NT>(P, T, tmem_base, stage, q, lane, c0, 4);
                    tc_fence_before();
                }
                __syncwarp();
                if (lane == 0) mb_arrive_first<CG>(&acc_empty[0]);
            }
        }
    } else if (warp == 2) {
        // ---------------- loader of the quantized columns ----------------
        const bool el = elect_one();
        uint32_t slot = 0, rph = 0;
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            const int vrows = max(0, min(MM_M, P.n_out - T.m0));
            for (int b = 0; b < n_blk && ok; b++) {
                ok &= mb_wait(&raw_empty[slot], rph ^ 1);
                uint8_t *dst = raw + (size_t)slot * C::RAW_SLOT;
                if (DT == LMOE_Q4_K) {
                    // one TMA tile load per projection
                    if (el) {
                        mb_expect_tx(&raw_full[slot], (uint32_t)C::RAW_SLOT);
#pragma unroll
                        for (int p = 0; p < NPROJ; p++)
                            tma_load_2d(dst + p * MM_M * Q4K_BYTES, &P.map[2 * T.sh + p], b * Q4K_BYTES, T.e * P.n_out + T.m0, &raw_full[slot]);
                    }
                } else if (P.lines) {
                    // 210-byte blocks start at any even address, and a row need not be a multiple of 16 bytes long, but 2^lg rows
                    // are: one tile load per row of a group of 2^lg takes that row's block of all groups, each
                    // inside a 240-byte window that starts on a 16-byte boundary.  (128 bulk copies of one window each
                    // cost 65 cycles apiece: 4180 cycles per stage; these at most eight loads keep ahead of the conversion.)
                    if (el) {
                        mb_expect_tx(&raw_full[slot], (uint32_t)C::RAW_SLOT);
                        for (int i = 0; i < 1 << P.lg; i++)
                            tma_load_2d(dst + (i << (7 - P.lg)) * GM_Q6_PITCH, &P.map[2 * T.sh], (i * row_bytes + b * Q6K_BYTES) & ~15,
                                        (T.e * P.n_out + T.m0) >> P.lg, &raw_full[slot]);
                    }
                } else {
                    // other row counts: each row's block inside its 224-byte aligned window (the last 16-byte granule holds
                    // at least one byte of the block, so the copy stays in mapped memory)
                    if (el) mb_expect_tx(&raw_full[slot], (uint32_t)vrows * GM_Q6_COPY);
                    __syncwarp();
                    const int64_t o0 = (int64_t)T.e * P.expert_bytes + (int64_t)T.m0 * row_bytes + b * Q6K_BYTES;
                    for (int r = lane; r < vrows; r += 32)
                        bulk_g2s(dst + gm_q6_line(r, P.lg) * GM_Q6_PITCH, P.w[T.sh] + ((o0 + (int64_t)r * row_bytes) & ~(int64_t)15),
                                 GM_Q6_COPY, &raw_full[slot]);
                }
                __syncwarp();
                if (++slot == C::RAW_SLOTS) { slot = 0; rph ^= 1; }
            }
        }
        landed(raw_full, C::RAW_SLOTS, slot, rph);
    } else if (NPROJ == 1 && warp == 1) {
        // ---------------- B loader: one bulk copy per 64-k block (the operand is stored in tile order) ----------------
        const bool el = elect_one();
        uint32_t slot = 0, ph = 0;
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            const int first = rank * gm_half<CG>(T.nv), brows = max(0, min(gm_half<CG>(T.nv), T.nv - first));
            const uint32_t bytes = (uint32_t)brows * 128u, grp = (uint32_t)gm_b_group<C::B_FULL, NT>(T.nv), sub = C::B_SLOT / grp;
            const uint8_t *src = P.xt + ((size_t)T.slot * k_blocks * NT + first) * 128;
            for (int kb = 0; kb < k_blocks && ok; kb += (int)grp) {
                ok &= mb_wait(&b_empty[slot], ph ^ 1);
                if (el) {
                    mb_expect_tx(&b_full[slot], bytes * grp);
                    for (uint32_t i = 0; i < grp && bytes; i++)
                        bulk_g2s(b_st + slot * C::B_SLOT + i * sub, src + (size_t)(kb + (int)i) * (NT * 128), bytes, &b_full[slot]);
                }
                __syncwarp();
                if (++slot == C::NB) { slot = 0; ph ^= 1; }
            }
        }
        landed(b_full, C::NB, slot, ph);
    } else if (NPROJ == 1 && CG == 2 && warp == 0 && rank == 1) {
        // ---------------- relay: a bulk copy signals its own CTA only; the issuer is told that this half of a slot has landed ----------------
        uint32_t slot = 0, ph = 0;
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            const int grp = gm_b_group<C::B_FULL, NT>(T.nv);
            for (int kb = 0; kb < k_blocks && ok; kb += grp) {
                ok &= mb_wait(&b_full[slot], ph);
                __syncwarp();
                if (lane == 0) mb_arrive_first<CG>(&b_full[slot]);
                if (++slot == C::NB) { slot = 0; ph ^= 1; }
            }
        }
    } else if (warp == 0 && rank == 0) {
        // ---------------- MMA issuer of the pair: the whole warp walks the loop, one elected lane issues ----------------
        // A wait that finds its barrier complete still takes over a hundred cycles beside the converting warps, two or three of
        // them more than a thin tile's multiplies.  So the next stage's barriers are asked, without waiting, before this stage's
        // multiplies are issued (512 tokens 514 -> 504 us, 1024 594 -> 581, op by op 512 849 -> 808).  The blocks of a ring slot are
        // a constant of the loop (there are up to three of it): with that and tc_mma_block, 512 tokens 475 -> 470, 1024 586 -> 579.
        const bool el = elect_one();
        const uint64_t bd0 = umma_desc(s32(b_st));
        const uint32_t blo = (uint32_t)bd0, bhi = (uint32_t)(bd0 >> 32), a0 = tmem_base + C::A_COL0;
        uint32_t it = 0, bs = 0, bph = 0, as = 0, aph = 0; // tiles; slot and phase of the B ring and of the operand stages
        bool b_here = false, a_here = false; // they were seen to be full
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step, it++) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            // (of one lane, so that the loop's operands are known to be the warp's)
            const int nv = __shfl_sync(0xffffffffu, T.nv, 0);
            const int npad = (nv + 15) & ~15;
            const uint32_t idesc = (1u << 4) | ((uint32_t)(npad >> 3) << 17) | ((uint32_t)(CG * MM_M >> 4) << 24);
            const uint32_t buf = NPROJ == 2 ? 0u : it & 1, cph = NPROJ == 2 ? it & 1 : (it >> 1) & 1;
            ok &= mb_wait(&acc_empty[buf], cph ^ 1);
            const uint32_t d = tmem_base + buf * NT;
            // k is a multiple of 256: a tile has a multiple of four 64-k blocks
            auto multiply = [&](auto group) {
                constexpr uint32_t GRP = decltype(group)::value, AB = C::A_BLKS, STEP = AB < GRP ? AB : GRP; // blocks between two waits
                uint32_t first = 1;
                for (int kb = 0; kb < k_blocks && ok; kb += 4) {
#pragma unroll
                    for (uint32_t u = 0; u < 4; u += STEP) {
                        if (C::NA * AB == 4) as = u / AB;
                        if (u % GRP == 0 && !b_here) ok &= mb_wait(&b_full[bs], bph);
                        if (u % AB == 0 && !a_here) ok &= mb_wait(&a_full[as], aph);
                        tc_fence_after();
                        const uint32_t a = a0 + C::A_COLS * as + (NPROJ == 2 ? 64u : 32u) * (u % AB);
                        const uint32_t bl = blo + bs * (C::B_SLOT >> 4) + u % GRP * ((C::B_SLOT >> 4) / GRP);
                        uint64_t *const b_done = &b_empty[bs], *const a_done = &a_empty[as];
                        const bool b_last = (u + STEP) % GRP == 0, a_last = (u + STEP) % AB == 0;
                        if (b_last) {
                            if (++bs == C::NB) { bs = 0; bph ^= 1; }
                            b_here = mb_test(&b_full[bs], bph);
                        }
                        if (a_last) {
                            if (++as == C::NA) { as = 0; aph ^= 1; }
                            a_here = mb_test(&a_full[as], aph);
                        }
                        if (el) {
#pragma unroll
                            for (uint32_t i = 0; i < STEP; i++)
                                tc_mma_block<CG, NPROJ == 2>(d, d + NT, a + (NPROJ == 2 ? 64u : 32u) * i, bl + i * ((C::B_SLOT >> 4) / GRP), bhi, idesc, u + i == 0 ? first : 0u);
                            if (b_last) tc_commit<CG>(b_done);
                            if (a_last) tc_commit<CG>(a_done);
                        }
                        __syncwarp();
                    }
                    first = 0;
                }
            };
            const int grp = gm_b_group<C::B_FULL, NT>(nv);
            if (grp == 4) multiply(std::integral_constant<uint32_t, 4>{});
            else if (C::B_FULL == 4) {}
            else if (grp == 2) multiply(std::integral_constant<uint32_t, 2>{});
            else if (C::B_FULL == 1) multiply(std::integral_constant<uint32_t, 1>{});
            if (el) tc_commit<CG>(&acc_full[buf]);
            __syncwarp();
        }
        // the last tile's commit covers all multiplies: none is in flight when the tensor memory is given back
        if (it) ok &= mb_wait(&acc_full[NPROJ == 2 ? 0u : (it - 1) & 1], NPROJ == 2 ? (it - 1) & 1 : ((it - 1) >> 1) & 1);
    } else if (NPROJ == 2 && warp >= 4) {
        // ---------------- B loaders: thread = (16-byte chunk of the 128-byte row piece, every 16th row) ----------------
        const int lt = tid - 128, ch = lt & 7, r0 = lt >> 3;
        const uint32_t dst0 = s32(b_st) + (uint32_t)(r0 * 128 + ((ch ^ (r0 & 7)) << 4));
        const uint32_t row16 = (uint32_t)(P.k >> 3); // 16-byte words of a row
        uint32_t slot = 0, ph = 0, done = 0, behind = 0; // ring slot and phase; oldest slot not yet announced, how many there are
        // A slot is announced two slots late: by then its copies have landed and the wait costs nothing.
        auto announce = [&]() {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mb_arrive_first<CG>(&b_full[done]);
            if (++done == C::NB) done = 0;
            behind--;
        };
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        constexpr int RPT = C::B_ROWS / 16; // rows of a thread
        int nsrc[RPT];
        auto brows = [&](const GmTile &N) { return min(gm_half<CG>(N.nv), N.nv - rank * gm_half<CG>(N.nv)); };
        auto rows = [&](const GmTile &N) {
            const int n = brows(N);
            const int32_t *src = P.src + N.slot * NT + rank * gm_half<CG>(N.nv);
#pragma unroll
            for (int i = 0; i < RPT; i++) nsrc[i] = r0 + 16 * i < n ? __ldg(src + r0 + 16 * i) : 0;
        };
        rows(next);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            uint32_t off[RPT];
#pragma unroll
            for (int i = 0; i < RPT; i++) off[i] = (uint32_t)nsrc[i] * row16 + ch;
            rows(next);
            const int n = brows(T);
            const int grp = gm_b_group<C::B_FULL, NT>(T.nv);
            const uint32_t sub = C::B_SLOT / grp;
            for (int kb = 0; kb < k_blocks && ok; kb += grp) {
                ok &= mb_wait(&b_empty[slot], ph ^ 1);
                for (int g = 0; g < grp; g++) {
                    const uint32_t dst = dst0 + slot * C::B_SLOT + g * sub;
                    const uint4 *base = reinterpret_cast<const uint4 *>(P.xt) + (size_t)(kb + g) * 8;
#pragma unroll
                    for (int i = 0; i < RPT; i++)
                        if (r0 + 16 * i < n)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 2048), "l"(base + off[i]) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (++slot == C::NB) { slot = 0; ph ^= 1; }
                if (++behind == 3) {
                    asm volatile("cp.async.wait_group 2;" ::: "memory");
                    announce();
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        while (behind > 0) announce();
    } else if (NPROJ == 1 && warp >= 4) {
        // ---------------- epilogue ----------------
        float *stage = reinterpret_cast<float *>(smem + C::O_EPI + (warp - 4) * C::EPI_BYTES);
        uint32_t it = 0;
        GmTile T, next = gm_tile<CG>(P, tile0, n_tiles, rank);
        for (int tile = tile0; tile < n_tiles && ok; tile += tile_step, it++) {
            T = next;
            next = gm_tile<CG>(P, tile + tile_step, n_tiles, rank);
            const uint32_t buf = it & 1;
            ok &= mb_wait(&acc_full[buf], (it >> 1) & 1);
            tc_fence_after();
            gm_epilogue<NPROJ, NT>(P, T, tmem_base + buf * NT, stage, warp & 3, lane, 0, 1);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive_first<CG>(&acc_empty[buf]);
        }
    }
    if (NPROJ == 1 && warp >= 4 && warp < GM_DQ0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (!ok && lane == 0) mm_timeout(P.flag, warp);
    tc_fence_before();
    __syncthreads();
    if (CG == 2) pair_sync(); // neither CTA leaves while the other may signal it or multiply its operands
    if (warp == 0) {
        if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

} // namespace

// ---- host side ---------------------------------------------------------------------------
// Routed rows per tile.  192 fills the tensor memory beside two accumulators with two operand stages and converts each
// weight least often; with fewer rows per expert every tile is thin whatever its limit, and lower tiles leave room for wide operand
// stages: two beside 128 rows, three beside 64.  A block's forward with its shared expert, evenly routed, cold L2, us with
// 64 / 128 / 192 by rows per expert:
//                              8                12                20                32                48                64                80
//   256 experts, 3072, 1024  380 / 386 / 409  415 / 404 / 429  447 / 447 / 476  568 / 526 / 548  748 / 640 / 689  861 / 726 / 697  1033 / 863 / 818
//   128 experts, 2048, 768   163 / 169 / 175  165 / 169 / 169  177 / 179 / 185  200 / 185 / 194  241 / 208 / 214  269 / 235 / 226  323 / 265 / 255
//   64 experts, 4096, 1536         -          263 / 269 / 279  269 / 273 / 290  277 / 283 / 298  349 / 298 / 314  403 / 327 / 331  466 / 380 / 357
//   64 experts, 2048, 512          -           93 / 95 / 97     93 / 93 / 98     99 / 97 / 101   116 / 101 / 107  124 / 110 / 112  142 / 128 / 120
//   16 experts, 4096, 2048         -                 -         136 / 142 / 144  138 / 146 / 150  167 / 148 / 159  206 / 157 / 161  216 / 189 / 167
// (Near the lines the tallest lists decide: how many of them just pass a tile's height.)
int mm_tile_rows(int64_t rows, int64_t n_expert) { return rows <= 20 * n_expert ? 64 : (rows <= 50 * n_expert ? 128 : 192); }

// Row tiles that `rows` routed rows over n_lists lists can make.
static int64_t mm_max_row_tiles(int64_t rows, int64_t n_lists, int nt) { return (rows + nt - 1) / nt + n_lists; }

bool mm_id_kernel_available(int dtype, int64_t n_out, int64_t k) {
    return (dtype == LMOE_Q4_K || dtype == LMOE_Q6_K) && n_out > 0 && k > 0 && k % QK_K == 0;
}

// Sizes and scratch of one grouped product: `rows` routed rows over n_expert lists, and `extra` rows of the shared expert.
MmRows mm_rows(int64_t rows, int64_t extra, int64_t n_expert) {
    MmRows R;
    R.rows = rows;
    R.extra = extra;
    R.n_expert = (int)n_expert;
    R.nt = mm_tile_rows(rows, n_expert);
    R.max_tiles = mm_max_row_tiles(rows, n_expert, R.nt) + (extra ? mm_max_row_tiles(extra, 1, R.nt) : 0);
    return R;
}
// Row tile table; its last 256 bytes hold the tile count.
size_t mm_tiles_bytes(const MmRows &R) { return lmoe_align_up((size_t)R.max_tiles * sizeof(int4), 256) + 256; }
// The tile-ordered f16 operand of width k.
size_t mm_tiled_bytes(const MmRows &R, int64_t k) { return lmoe_align_up((size_t)R.max_tiles * (size_t)(k / MM_K) * R.nt * 128, 256); }

// Source rows of the tile rows (stage_rows_kernel).
size_t mm_src_bytes(const MmRows &R) { return lmoe_align_up((size_t)R.max_tiles * R.nt * 4, 256); }

static int32_t *mm_tile_count(const MmRows &R, void *tiles_ws) {
    return reinterpret_cast<int32_t *>(static_cast<uint8_t *>(tiles_ws) + mm_tiles_bytes(R) - 256);
}

// Row tiles from the per-expert counts, then the operand in tile order.  pos / spos / sfid (each may be NULL): position in
// tile order and in expert-sorted order of every flat id, flat id of every sorted row; the shared expert's rows have the
// flat ids rows, rows + 1, ...
lmoe_status launch_gather_tiles(const MmRows &R, const void *x, int x_f16, int x_per_row, int top_k, int k, const uint32_t *tpe,
                                const int32_t *ids_map, int64_t map_stride, void *tiles_ws, void *xt, int32_t *pos, int32_t *spos,
                                int32_t *sfid, cudaStream_t s) {
    if (R.n_expert > 512) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "grouped GEMM supports at most 512 experts");
    int4 *tiles = static_cast<int4 *>(tiles_ws);
    int32_t *n_tiles = mm_tile_count(R, tiles_ws);
    launch_pdl(row_tiles_kernel, 1, 1024, 0, s, tpe, R.n_expert, (int)R.extra, R.nt, tiles, n_tiles, (int)R.max_tiles);
    LMOE_LAUNCH_CHECK("row_tiles_kernel");
    const dim3 grid((unsigned)R.max_tiles, (unsigned)((R.nt + GT_ROWS - 1) / GT_ROWS));
    if (x_f16)
        launch_pdl(gather_tiles_kernel<true>, grid, 256, 0, s, x, x_per_row, top_k, k, tiles, n_tiles, ids_map, (int)map_stride, R.n_expert,
                                                       (int)R.rows, R.nt, static_cast<uint8_t *>(xt), pos, spos, sfid);
    else
        launch_pdl(gather_tiles_kernel<false>, grid, 256, 0, s, x, x_per_row, top_k, k, tiles, n_tiles, ids_map, (int)map_stride, R.n_expert,
                                                        (int)R.rows, R.nt, static_cast<uint8_t *>(xt), pos, spos, sfid);
    LMOE_LAUNCH_CHECK("gather_tiles_kernel");
    return LMOE_OK;
}

// The same tables for the gate/up kernel: x as f16 in token order (`xh`, x_rows rows of k values) and the source row of every
// tile row (`src`, mm_src_bytes).
lmoe_status launch_stage_rows(const MmRows &R, const void *x, int x_f16, int64_t x_rows, int top_k, int k, const uint32_t *tpe,
                              const int32_t *ids_map, int64_t map_stride, void *tiles_ws, void *xh, int32_t *src, int32_t *pos,
                              int32_t *spos, int32_t *sfid, cudaStream_t s) {
    if (R.n_expert > 512) return lmoe_fail(LMOE_ERR_UNSUPPORTED, "grouped GEMM supports at most 512 experts");
    int4 *tiles = static_cast<int4 *>(tiles_ws);
    int32_t *n_tiles = mm_tile_count(R, tiles_ws);
    launch_pdl(row_tiles_kernel, 1, 1024, 0, s, tpe, R.n_expert, (int)R.extra, R.nt, tiles, n_tiles, (int)R.max_tiles);
    LMOE_LAUNCH_CHECK("row_tiles_kernel");
    const int64_t chunks = x_rows * (k / 8);
    const int conv = (int)((chunks + 255) / 256);
    const unsigned grid = (unsigned)(conv + R.max_tiles);
    if (x_f16)
        launch_pdl(stage_rows_kernel<true>, grid, 256, 0, s, x, chunks, conv, top_k, tiles, n_tiles, ids_map, (int)map_stride, R.n_expert,
                                                     (int)R.rows, R.nt, static_cast<uint8_t *>(xh), src, pos, spos, sfid);
    else
        launch_pdl(stage_rows_kernel<false>, grid, 256, 0, s, x, chunks, conv, top_k, tiles, n_tiles, ids_map, (int)map_stride, R.n_expert,
                                                      (int)R.rows, R.nt, static_cast<uint8_t *>(xh), src, pos, spos, sfid);
    LMOE_LAUNCH_CHECK("stage_rows_kernel");
    return LMOE_OK;
}

// A 2-D TMA view [rows][row_elems], boxes of box_elems x box_rows.  The encoder is a driver entry point, fetched through
// the runtime (no link against the driver library).
static lmoe_status make_map_2d(CUtensorMap *map, CUtensorMapDataType type, int elem_bytes, const void *base, uint64_t row_elems,
                               uint64_t rows, uint32_t box_elems, uint32_t box_rows) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static encode_fn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
            q != cudaDriverEntryPointSuccess)
            return lmoe_fail(LMOE_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
        encode = reinterpret_cast<encode_fn>(fn);
    }
    const uint64_t row_bytes = row_elems * elem_bytes;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) || row_bytes % 16 || box_elems * elem_bytes % 16 || box_elems > 256 || box_rows > 256)
        return lmoe_fail(LMOE_ERR_UNSUPPORTED, "buffer layout does not fit a TMA tile (16-byte alignment of base, row and box)");
    const cuuint64_t dims[2] = {row_elems, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_elems, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc = encode(map, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return lmoe_fail(LMOE_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)rc);
    return LMOE_OK;
}
static lmoe_status make_rows_map(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes,
                                 uint32_t box_rows) {
    return make_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, base, row_bytes, rows, box_bytes, box_rows);
}

// st / sh: the stacks of the one or two projections, of the experts and (NULL without extra rows) of the shared expert.
template <int DT, int NPROJ, int NT, int CG>
static lmoe_status launch_grouped(const MmRows &R, const lmoe_expert_stack *const (&st)[2], const lmoe_expert_stack *const (&sh)[2],
                                  const void *xt, const int32_t *src, const int32_t *ids_map, int64_t map_stride, const float *row_scale,
                                  float *out, int sorted, void *tiles_ws, uint32_t *flag, cudaStream_t stream) {
    using C = GmCfg<DT, NPROJ, NT, CG>;
    GmParams P;
    P.lg = gm_q6_lg((int)(st[0]->k / QK_K));
    P.lines = (st[0]->n_out & ((1 << P.lg) - 1)) == 0;
    for (int p = 0; p < 2 * NPROJ; p++) {
        const lmoe_expert_stack *s = p < NPROJ ? st[p] : sh[p - NPROJ];
        if (!s) continue;
        CUtensorMap *map = &P.map[2 * (p / NPROJ) + p % NPROJ];
        lmoe_status mst = LMOE_OK;
        if (DT == LMOE_Q4_K)
            mst = make_rows_map(map, s->blocks(), (uint64_t)s->row_bytes(), (uint64_t)s->n_expert * s->n_out, Q4K_BYTES, MM_M);
        else if (P.lines)
            mst = make_rows_map(map, s->blocks(), (uint64_t)s->row_bytes() << P.lg, (uint64_t)(s->n_expert * s->n_out) >> P.lg, GM_Q6_PITCH, MM_M >> P.lg);
        if (mst) return mst;
    }
    P.w[0] = st[0]->blocks();
    P.w[1] = sh[0] ? sh[0]->blocks() : nullptr;
    P.expert_bytes = st[0]->expert_bytes(); P.n_out = (int)st[0]->n_out; P.k = (int)st[0]->k;
    P.n_expert = R.n_expert; P.m_tiles = (int)((st[0]->n_out + CG * MM_M - 1) / (CG * MM_M));
    P.xt = static_cast<const uint8_t *>(xt); P.src = src; P.ids_map = ids_map; P.map_stride = (int)map_stride;
    P.tiles = static_cast<const int4 *>(tiles_ws); P.n_tiles = mm_tile_count(R, tiles_ws);
    P.row_scale = row_scale; P.out = out; P.sorted = sorted; P.flag = flag;
    P.vec = st[0]->n_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    if (NPROJ == 1 && sorted && P.vec) {
        lmoe_status mst = make_map_2d(&P.map_out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, out, (uint64_t)st[0]->n_out, (uint64_t)(R.rows + R.extra),
                                      32, GM_BOX_ROWS);
        if (mst) return mst;
    }
    auto kernel = grouped_mm_kernel<DT, NPROJ, NT, CG>;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GM_THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = stream;
    cfg.attrs = attr;
    // The launch (barriers, tensor memory, the pair's meeting) overlaps the end of the kernel before.  Plain against so, a layer of 8
    // experts of 256, 400 / 1228 / 3000 tokens: 61.7 / 69.9 / 96.5 us, 56.3 / 67.6 / 92.2; 64 of 512, 640 / 3000 tokens: 127 / 305,
    // 122 / 299; a single product of 8 experts [3072 x 1024], 256 tokens: 24.7, 22.7.  From 2048 tokens of the large layers on the two
    // differ by less than two runs of one of them.
    cfg.numAttrs = 2;
    static thread_local int c_dev = -1, c_grid = 0;
    int dev = 0;
    LMOE_CUDA(cudaGetDevice(&dev));
    if (dev != c_dev) {
        int sms = 0, pairs = 0;
        LMOE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        LMOE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        cfg.gridDim = dim3((unsigned)(sms / CG * CG));
        LMOE_CUDA(cudaOccupancyMaxActiveClusters(&pairs, kernel, &cfg));
        if (pairs < 1) return lmoe_fail(LMOE_ERR_CUDA, "no place for a tile's CTAs");
        c_grid = CG * pairs < sms ? CG * pairs : sms / CG * CG;
        c_dev = dev;
    }
    cfg.gridDim = dim3((unsigned)c_grid);
    LMOE_CUDA(cudaLaunchKernelEx(&cfg, kernel, P));
    LMOE_LAUNCH_CHECK("grouped_mm_kernel");
    return LMOE_OK;
}

// Up to this many blocks of 128 weight rows, an odd number of them goes to single CTAs: a pair's tile is two blocks high, and the
// second CTA of the last one would convert rows of no use.  Q4_K, pairs against single CTAs: 512 tokens, ten of 256 experts
// [128 x 1024] 37.1 us against 28.9, [128 x 3072] 58.2 / 42.0, [640 x 3072] 119 / 109; 64 experts, 8 a token, [1152 x 1024] 37.0 / 32.9;
// Q6_K, 8192 rows of 4 experts, [384 x 1024] 37.0 / 29.0, [1664 x 1024] 67.7 / 60.5.  Where both take as many rounds over the SMs, long rows
// in pairs are up to 10 % shorter ([1152 x 3072] of 4 experts 81.2 / 90.0); from 17 blocks on that is the rule ([2176 x 3072] of 64
// experts 102 / 107).
constexpr int GM_SINGLE_BLOCKS = 13;

// One grouped projection on the row tiles that launch_gather_tiles made (`xt`: the f16 operand in tile order; `flag`: 4 device
// words, zero = clean).  Rows of `out` by flat id, times row_scale when given, or (`sorted`) unscaled in expert-sorted order.
lmoe_status launch_mm_id(const MmRows &R, const lmoe_expert_stack *st, const lmoe_expert_stack *shared, const void *xt,
                         const int32_t *ids_map, int64_t map_stride, const float *row_scale, float *out, int sorted, void *tiles_ws,
                         uint32_t *flag, cudaStream_t stream) {
    const int64_t blocks = (st->n_out + MM_M - 1) / MM_M;
    if ((blocks & 1) && blocks <= GM_SINGLE_BLOCKS) {
        auto fn = R.nt == 64 ? (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 64, 1> : launch_grouped<LMOE_Q6_K, 1, 64, 1>)
                  : R.nt == 128 ? (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 128, 1> : launch_grouped<LMOE_Q6_K, 1, 128, 1>)
                              : (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 192, 1> : launch_grouped<LMOE_Q6_K, 1, 192, 1>);
        return fn(R, {st, nullptr}, {shared, nullptr}, xt, nullptr, ids_map, map_stride, row_scale, out, sorted, tiles_ws, flag, stream);
    }
    auto fn = R.nt == 64 ? (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 64, 2> : launch_grouped<LMOE_Q6_K, 1, 64, 2>)
              : R.nt == 128 ? (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 128, 2> : launch_grouped<LMOE_Q6_K, 1, 128, 2>)
                          : (st->dtype == LMOE_Q4_K ? launch_grouped<LMOE_Q4_K, 1, 192, 2> : launch_grouped<LMOE_Q6_K, 1, 192, 2>);
    return fn(R, {st, nullptr}, {shared, nullptr}, xt, nullptr, ids_map, map_stride, row_scale, out, sorted, tiles_ws, flag, stream);
}

// gate and up in one kernel, SwiGLU applied: act[rows, ff] (f32), rows by flat id or in expert-sorted order.
lmoe_status launch_mm_gateup(const MmRows &R, const lmoe_expert_stack *gate, const lmoe_expert_stack *up, const lmoe_expert_stack *sh_gate,
                             const lmoe_expert_stack *sh_up, const void *xh, const int32_t *src, const int32_t *ids_map, int64_t map_stride, float *act,
                             int sorted, void *tiles_ws, uint32_t *flag, cudaStream_t stream) {
    if (gate->dtype != LMOE_Q4_K || up->dtype != LMOE_Q4_K)
        return lmoe_fail(LMOE_ERR_UNSUPPORTED, "the fused gate/up kernel is built for Q4_K stacks");
    auto fn = R.nt == 64 ? launch_grouped<LMOE_Q4_K, 2, 64, 2> : R.nt == 128 ? launch_grouped<LMOE_Q4_K, 2, 128, 2> : launch_grouped<LMOE_Q4_K, 2, 192, 2>;
    return fn(R, {gate, up}, {sh_gate, sh_up}, xh, src, ids_map, map_stride, nullptr, act, sorted, tiles_ws, flag, stream);
}
