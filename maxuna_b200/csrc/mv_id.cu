// Stand-alone indexed quantized mat-vec: out[t,s,:] = W[ids[t,s]] . x[t, s|0, :].
// Reference: `ops::mul_mv_id`, src/ops/mv_id.rs:37-45; kernels
// kernel_mul_mv_id_q{4,6}_K_f32_v, src/ops/mv.metal:181-290, 413-504, 638-717.
//
// Four kernels.  Three carry the activations as four signed base-256 digits of 30-bit integers under a power of two per
// 256-wide block, and multiply them with the raw 4- and 6-bit fields on the integer tensor-core path (mma.sync u8 x s8 -> s32,
// exact), as the fused decode kernel does; the scales come in once per super-block.  The integers hold every value within 2^6
// of the block's largest exactly and the others to 2^-30 of it, so a product is no further from 64 bits than one of f32
// values and sums (relative error Q4_K 0.6e-7 to 1.4e-7 against 1.7e-7 to 2.9e-7, Q6_K 0.6e-7 to 0.8e-7 against 0.8e-7 to
// 1.0e-7, for normal and log-normal values, products of two, and one value of a block or row 100 or 10^4 times the others;
// three digits, 24 bits under the largest magnitude: up to 13e-7, and NaN below 2.5e-32).
// A lane-per-16-bytes f32 dot product is bound by its conversions and multiply-adds, but has nothing to set up:
//   mv_row_kernel    f32 activations and sums, a warp per row: little work, few rows, and Q6_K rows that the ring does not
//                    take (see mv_rows_better).
// The others:
//   mv_expert_kernel the ordinary case, bound by the weight stream: pairs of the same expert share a pass over its rows, which
//                    come through shared memory in bulk copies.  Weights of 3 / 16 / 64 tokens with ten experts each, against
//                    mv_pair_kernel: [1024 x 3072] Q4_K 17 / 78 / 290 -> 15 / 55 / 144 us, [3072 x 1024] Q6_K (whose 210-byte
//                    super-blocks cost two loads a word from global memory) 39 / 203 / 810 -> 21 / 84 / 221 us.
//   mv_pair_kernel   Q4_K of any shape, one (token, slot) pair per block row; what is left to it are rows too long for the
//                    ring.  Weights go straight from global memory into the A fragments.
//   mv_multi_kernel  many pairs of ONE weight matrix (the shared expert, a plain matrix): eight pairs are the columns of
//                    an MMA, so a super-block is unpacked once for 32 pairs.  512 pairs of [1024 x 3072] Q4_K: 816 -> 68 us.
//                    From where it is the shorter one, mv_dense.cu serves these.
#include <cooperative_groups.h>
#include "common.cuh"
#include "mv_digits.cuh"
#include "stream_math.cuh"

namespace {

constexpr int MV_THREADS = 256, MV_ROWS = 64; // rows of a block: four MMA row tiles, the K dimension in two halves
// ---- raw fields of two rows of one super-block, as this lane's part of the MMA A fragments --------------------------
// Q4_K: bytes 8t .. 8t+7 of each 32-byte run (low nibbles: sub-block 2j, high: 2j+1), and the 16-byte header.
struct MvQ4 {
    uint4 hg, hG;
    uint2 wg[4], wG[4];
    __device__ __forceinline__ void load(const uint8_t *bg, const uint8_t *bG, int t) {
        hg = __ldg(reinterpret_cast<const uint4 *>(bg));
        hG = __ldg(reinterpret_cast<const uint4 *>(bG));
#pragma unroll
        for (int j = 0; j < 4; j++) {
            wg[j] = __ldg(reinterpret_cast<const uint2 *>(bg + 16 + 32 * j + 8 * t));
            wG[j] = __ldg(reinterpret_cast<const uint2 *>(bG + 16 + 32 * j + 8 * t));
        }
    }
};
// Four bytes at an even address: the one or two aligned words that hold them (never a word without a byte of them).
__device__ __forceinline__ uint32_t ldg_a2(const uint8_t *p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t lo = __ldg(q), hi = __ldg(q + ((a >> 1) & 1));
    return __byte_perm(lo, hi, (a & 2) ? 0x5432u : 0x3210u);
}
// Q6_K: word 4t .. 4t+3 of every 16-wide run of ql (four per half) and qh (two per half), the sixteen scales, d.
struct MvQ6 {
    uint32_t qg[8], qG[8], hg[4], hG[4], sg[4], sG[4];
    float dg, dG;
    __device__ __forceinline__ void load(const uint8_t *bg, const uint8_t *bG, int t) {
#pragma unroll
        for (int i = 0; i < 8; i++) { // ql run i: half i / 4, 16-wide range i % 4
            qg[i] = ldg_a2(bg + 16 * i + 4 * t);
            qG[i] = ldg_a2(bG + 16 * i + 4 * t);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            hg[i] = ldg_a2(bg + 128 + 16 * i + 4 * t);
            hG[i] = ldg_a2(bG + 128 + 16 * i + 4 * t);
            sg[i] = ldg_a2(bg + 192 + 4 * i);
            sG[i] = ldg_a2(bG + 192 + 4 * i);
        }
        dg = lmoe_h2f(__ldg(reinterpret_cast<const uint16_t *>(bg + 208)));
        dG = lmoe_h2f(__ldg(reinterpret_cast<const uint16_t *>(bG + 208)));
    }
};

// A fragments of one super-block: MMAs of the integer product (8 of k = 32 for Q4_K, 16 of k = 16 for Q6_K), the integer
// scale of each, and the fragments of the one f16 product that carries the Q4_K mins / the Q6_K "-32".
template <int DT>
struct MvA;
template <>
struct MvA<LMOE_Q4_K> {
    static constexpr int N = 8;
    uint32_t a[N][4], f[4];
    uint32_t scg[2], scG[2];
    float dg, dG, mg, mG; // factors of the integer product and of the f16 product
    __device__ __forceinline__ void unpack(const MvQ4 &R, int t) {
        constexpr uint32_t M4 = 0x0F0F0F0Fu;
        uint32_t mng[2], mnG[2];
        q4k_unpack_scales(R.hg.y, R.hg.z, R.hg.w, scg[0], scg[1], mng[0], mng[1]);
        q4k_unpack_scales(R.hG.y, R.hG.z, R.hG.w, scG[0], scG[1], mnG[0], mnG[1]);
        dg = lmoe_h2f((uint16_t)(R.hg.x & 0xffff));
        dG = lmoe_h2f((uint16_t)(R.hG.x & 0xffff));
        // the six-bit mins enter the f16 product as subnormals (times 2^-24)
        mg = lmoe_h2f((uint16_t)(R.hg.x >> 16)) * (16777216.f * MV_SUM_UNSCALE);
        mG = lmoe_h2f((uint16_t)(R.hG.x >> 16)) * (16777216.f * MV_SUM_UNSCALE);
        const uint32_t sel = (t & 1) ? 0x4342u : 0x4140u;
        f[0] = __byte_perm(t < 2 ? mng[0] : mng[1], 0u, sel);
        f[1] = __byte_perm(t < 2 ? mnG[0] : mnG[1], 0u, sel);
        f[2] = f[3] = 0u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            a[2 * j][0] = R.wg[j].x & M4; a[2 * j][1] = R.wG[j].x & M4; a[2 * j][2] = R.wg[j].y & M4; a[2 * j][3] = R.wG[j].y & M4;
            a[2 * j + 1][0] = (R.wg[j].x >> 4) & M4; a[2 * j + 1][1] = (R.wG[j].x >> 4) & M4;
            a[2 * j + 1][2] = (R.wg[j].y >> 4) & M4; a[2 * j + 1][3] = (R.wG[j].y >> 4) & M4;
        }
    }
    __device__ __forceinline__ int sg(int i) const { return ubyte(scg[i >> 2], i & 3); }
    __device__ __forceinline__ int sG(int i) const { return ubyte(scG[i >> 2], i & 3); }
    __device__ __forceinline__ void mma(int i, int (&d)[4], const int8_t *x, int t) const {
        const uint2 b = *reinterpret_cast<const uint2 *>(x + 32 * i + 8 * t);
        imma16832_z(d, a[i][0], a[i][1], a[i][2], a[i][3], b.x, b.y);
    }
};
template <>
struct MvA<LMOE_Q6_K> {
    static constexpr int N = 16;
    uint32_t a[N][2], f[4];
    uint32_t scg[4], scG[4];
    float dg, dG, mg, mG;
    __device__ __forceinline__ void unpack(const MvQ6 &R, int t) {
        constexpr uint32_t M4 = 0x0F0F0F0Fu, M2 = 0x30303030u;
#pragma unroll
        for (int q = 0; q < 4; q++) { scg[q] = R.sg[q]; scG[q] = R.sG[q]; }
        dg = R.dg; dG = R.dG;
        mg = dg * MV_OFFSET;
        mG = dG * MV_OFFSET;
        // scales 2t, 2t+1 and 2t+8, 2t+9 of each row, as f16 pairs
        auto pair = [&](const uint32_t (&s)[4], int w) {
            const uint32_t v = t >= 2 ? s[2 * w + 1] : s[2 * w];
            const __half2 h = __floats2half2_rn((float)sbyte(v, 2 * (t & 1)), (float)sbyte(v, 2 * (t & 1) + 1));
            return *reinterpret_cast<const uint32_t *>(&h);
        };
        f[0] = pair(scg, 0); f[1] = pair(scG, 0); f[2] = pair(scg, 1); f[3] = pair(scG, 1);
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    // sub-block 8 n + 2 i + c: group i (nibble i / 2 of ql run 2 (i & 1) + c, bits 2 i of qh run c)
                    const uint32_t qg = R.qg[4 * n + 2 * (i & 1) + c], qG = R.qG[4 * n + 2 * (i & 1) + c], hg = R.hg[2 * n + c], hG = R.hG[2 * n + c];
                    const uint32_t lg = (i & 2) ? qg >> 4 : qg, lG = (i & 2) ? qG >> 4 : qG;
                    const uint32_t ug = i == 0 ? hg << 4 : (i == 1 ? hg << 2 : (i == 2 ? hg : hg >> 2));
                    const uint32_t uG = i == 0 ? hG << 4 : (i == 1 ? hG << 2 : (i == 2 ? hG : hG >> 2));
                    a[8 * n + 2 * i + c][0] = (lg & M4) | (ug & M2);
                    a[8 * n + 2 * i + c][1] = (lG & M4) | (uG & M2);
                }
    }
    __device__ __forceinline__ int sg(int i) const { return sbyte(scg[i >> 2], i & 3); }
    __device__ __forceinline__ int sG(int i) const { return sbyte(scG[i >> 2], i & 3); }
    __device__ __forceinline__ void mma(int i, int (&d)[4], const int8_t *x, int t) const {
        imma16816_z(d, a[i][0], a[i][1], *reinterpret_cast<const uint32_t *>(x + 16 * i + 4 * t));
    }
};
template <int DT> struct MvRaw;
template <> struct MvRaw<LMOE_Q4_K> { typedef MvQ4 T; };
template <> struct MvRaw<LMOE_Q6_K> { typedef MvQ6 T; };

// d += a * b (f16 inputs)
__device__ __forceinline__ void mma16816_acc(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int MV_PAIR_BLOCKS = 32; // super-blocks of the activation row staged at a time (8192 values)

// ---- a warp per row -------------------------------------------------------------------
// grid (ceil(n_out / 8), pairs): lanes stride over 16-byte pieces of the row, decode in registers, multiply f32 activations.
constexpr int MR_WARPS = 4, MR_ROWS = 2; // rows of a warp

__device__ __forceinline__ float dot_row_q4k(const uint8_t *__restrict__ row, const float *__restrict__ x, int nb, int lane) {
    float acc = 0.f;
    for (int u = lane; u < nb * 8; u += 32) {
        const int b = u >> 3, c = u & 7, j = c >> 1, h = c & 1;
        const uint8_t *blk = row + (size_t)b * Q4K_BYTES;
        const uint32_t dm = __ldg(reinterpret_cast<const uint32_t *>(blk));
        const float d = lmoe_h2f((uint16_t)(dm & 0xffff)), dmin = lmoe_h2f((uint16_t)(dm >> 16));
        int sc0, mn0, sc1, mn1;
        q4k_scale_min(blk + 4, 2 * j, sc0, mn0);
        q4k_scale_min(blk + 4, 2 * j + 1, sc1, mn1);
        const uint4 qv = __ldg(reinterpret_cast<const uint4 *>(blk + 16 + 16 * c));
        const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w};
        const float *xl = x + b * QK_K + 64 * j + 16 * h, *xh = xl + 32;
        float slo = 0.f, shi = 0.f, xsl = 0.f, xsh = 0.f;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(xl + 4 * w)), g = __ldg(reinterpret_cast<const float4 *>(xh + 4 * w));
            const uint32_t q = qw[w];
            slo += a.x * (float)(q & 15) + a.y * (float)((q >> 8) & 15) + a.z * (float)((q >> 16) & 15) + a.w * (float)((q >> 24) & 15);
            shi += g.x * (float)((q >> 4) & 15) + g.y * (float)((q >> 12) & 15) + g.z * (float)((q >> 20) & 15) + g.w * (float)(q >> 28);
            xsl += a.x + a.y + a.z + a.w;
            xsh += g.x + g.y + g.z + g.w;
        }
        acc += d * ((float)sc0 * slo + (float)sc1 * shi) - dmin * ((float)mn0 * xsl + (float)mn1 * xsh);
    }
    return acc;
}

__device__ __forceinline__ float dot_row_q6k(const uint8_t *__restrict__ row, const float *__restrict__ x, int nb, int lane) {
    float acc = 0.f;
    for (int u = lane; u < nb * 16; u += 32) {
        const int b = u >> 4, n = (u >> 3) & 1, lg = u & 7;
        const uint8_t *blk = row + (size_t)b * Q6K_BYTES;
        const uint32_t qa = ld_u32_unaligned2(blk + 64 * n + 4 * lg), qb = ld_u32_unaligned2(blk + 64 * n + 32 + 4 * lg);
        const uint32_t qh = ld_u32_unaligned2(blk + 128 + 32 * n + 4 * lg);
        const int8_t *sc = reinterpret_cast<const int8_t *>(blk + 192) + 8 * n + (lg >> 2);
        const float d = lmoe_h2f(*reinterpret_cast<const uint16_t *>(blk + 208));
        const float *xp = x + b * QK_K + 128 * n + 4 * lg;
        float xa[4][4], s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(xp + 32 * g));
            xa[g][0] = v.x; xa[g][1] = v.y; xa[g][2] = v.z; xa[g][3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int h = (qh >> (8 * i)) & 0xff, a = (qa >> (8 * i)) & 0xff, c = (qb >> (8 * i)) & 0xff;
            s[0] += xa[0][i] * (float)(((a & 15) | ((h & 3) << 4)) - 32);
            s[1] += xa[1][i] * (float)(((c & 15) | (((h >> 2) & 3) << 4)) - 32);
            s[2] += xa[2][i] * (float)(((a >> 4) | (((h >> 4) & 3) << 4)) - 32);
            s[3] += xa[3][i] * (float)(((c >> 4) | (((h >> 6) & 3) << 4)) - 32);
        }
        acc += d * ((float)sc[0] * s[0] + (float)sc[2] * s[1] + (float)sc[4] * s[2] + (float)sc[6] * s[3]);
    }
    return acc;
}

template <int DT>
__global__ void __launch_bounds__(MR_WARPS * 32)
mv_row_kernel(const uint8_t *__restrict__ w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *__restrict__ x,
              int x_per_row, const uint32_t *__restrict__ ids, int top_k, float *__restrict__ out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pair = blockIdx.y, nb = k / QK_K;
    const uint32_t e = ids ? ids[pair] : 0u;
    const int64_t row_bytes = (int64_t)nb * (DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES);
    const float *xr = x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k;
    const int r0 = (blockIdx.x * MR_WARPS + warp) * MR_ROWS;
#pragma unroll
    for (int r = 0; r < MR_ROWS; r++) {
        if (r0 + r >= n_out) break;
        float v = 0.f;
        if (e < (uint32_t)n_expert) { // an out-of-range id produces a zero row
            const uint8_t *row = w + (size_t)e * expert_bytes + (size_t)(r0 + r) * row_bytes;
            v = DT == LMOE_Q4_K ? dot_row_q4k(row, xr, nb, lane) : dot_row_q6k(row, xr, nb, lane);
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (lane == 0) out[(size_t)pair * n_out + r0 + r] = v;
    }
}

// ---- one pair -------------------------------------------------------------------------
// grid (ceil(n_out / 64), pairs), eight warps: row tile = warp % 4, K half = warp / 4.
// MMA columns 0-3: the digits; 4-7 repeat column 0 and are not read.
template <int DT>
__global__ void __launch_bounds__(MV_THREADS, 2)
mv_pair_kernel(const uint8_t *__restrict__ w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *__restrict__ x,
               int x_per_row, const uint32_t *__restrict__ ids, int top_k, float *__restrict__ out) {
    pdl_begin();
    constexpr int SUB = DT == LMOE_Q4_K ? 32 : 16, NS = QK_K / SUB;
    constexpr int TS = DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES;
    extern __shared__ __align__(16) uint8_t mv_smem[];
    __shared__ float red[2][MV_ROWS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int pair = blockIdx.y, nb = k / QK_K;
    const int64_t row_bytes = (int64_t)nb * TS;
    const uint32_t e = ids ? ids[pair] : 0u;
    const int r_base = blockIdx.x * MV_ROWS;
    if (e >= (uint32_t)n_expert) { // an out-of-range id produces a zero row
        if (tid < MV_ROWS && r_base + tid < n_out) out[(size_t)pair * n_out + r_base + tid] = 0.f;
        return;
    }
    const int bc = min(nb, MV_PAIR_BLOCKS), pitch = bc * QK_K + 32; // super-blocks staged at a time, bytes of a digit column
    int8_t *xc = reinterpret_cast<int8_t *>(mv_smem);
    __half *sh = reinterpret_cast<__half *>(mv_smem + MV_NDIG * pitch);
    float *sxs = reinterpret_cast<float *>(mv_smem + MV_NDIG * pitch + MV_PARTS * bc * NS * 2);
    const int rt = warp & 3, ks = warp >> 2;
    const int rg = min(r_base + 16 * rt + g, n_out - 1), rG = min(r_base + 16 * rt + g + 8, n_out - 1);
    const uint8_t *wb = w + (size_t)e * expert_bytes;
    const uint8_t *pg = wb + (size_t)rg * row_bytes, *pG = wb + (size_t)rG * row_bytes;
    const float *xr = x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k;
    const int8_t *xcol = xc + (g < MV_NDIG ? g : 0) * pitch;
    const __half *scol = sh + (g < MV_PARTS ? g : 0) * bc * NS; // columns 0-2: the parts of the sums
    float yg = 0.f, yG = 0.f;
    for (int c0 = 0; c0 < nb; c0 += bc) {
        const int bn = min(bc, nb - c0);
        typename MvRaw<DT>::T raw;
        if (ks < bn) raw.load(pg + (size_t)(c0 + ks) * TS, pG + (size_t)(c0 + ks) * TS, t); // on its way while the activations are staged
        if (c0) __syncthreads(); // the previous digits have been read
        for (int b = warp; b < bn; b += MV_THREADS / 32) {
            uint2 dig[MV_NDIG];
            float sx;
            __half part[MV_PARTS];
            MvX in;
            in.load(xr + (size_t)(c0 + b) * QK_K, true, lane);
            mv_digits<SUB>(in, dig, sx, part);
#pragma unroll
            for (int d = 0; d < MV_NDIG; d++) *reinterpret_cast<uint2 *>(xc + d * pitch + b * QK_K + lane * 8) = dig[d];
            if ((lane & (SUB / 8 - 1)) == 0) {
#pragma unroll
                for (int h = 0; h < MV_PARTS; h++) sh[(h * bc + b) * NS + lane / (SUB / 8)] = part[h];
            }
            if (lane == 0) sxs[b] = sx;
        }
        __syncthreads();
        for (int b = ks; b < bn; b += 2) {
            MvA<DT> A;
            A.unpack(raw, t);
            if (b + 2 < bn) raw.load(pg + (size_t)(c0 + b + 2) * TS, pG + (size_t)(c0 + b + 2) * TS, t);
            float cm[4] = {0.f, 0.f, 0.f, 0.f};
            const uint32_t s0 = *reinterpret_cast<const uint32_t *>(scol + b * NS + 2 * t);
            const uint32_t s1 = NS == 16 ? *reinterpret_cast<const uint32_t *>(scol + b * NS + 2 * t + 8) : 0u;
            mma16816_acc(cm, A.f, s0, s1);
            int al[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < MvA<DT>::N; i++) {
                int f[4];
                A.mma(i, f, xcol + b * QK_K, t);
                const int sg = A.sg(i), sG = A.sG(i);
                al[0] += sg * f[0]; al[1] += sg * f[1]; al[2] += sG * f[2]; al[3] += sG * f[3];
            }
            // lane t = 0 holds columns 0, 1, lane t = 1 columns 2, 3 (no part of the sums in 3)
            const float f0 = t == 0 ? 16777216.f : (t == 1 ? 256.f : 0.f), f1 = t == 0 ? 65536.f : (t == 1 ? 1.f : 0.f), sx = sxs[b];
            const float m0 = t < 2 ? 1.f : 0.f, m1 = t == 0 ? 1.f : 0.f;
            yg += sx * (A.dg * (f0 * (float)al[0] + f1 * (float)al[1]) - A.mg * (m0 * cm[0] + m1 * cm[1]));
            yG += sx * (A.dG * (f0 * (float)al[2] + f1 * (float)al[3]) - A.mG * (m0 * cm[2] + m1 * cm[3]));
        }
    }
    yg += __shfl_xor_sync(0xffffffffu, yg, 1);
    yG += __shfl_xor_sync(0xffffffffu, yG, 1);
    if (t == 0) {
        red[ks][16 * rt + g] = yg;
        red[ks][16 * rt + g + 8] = yG;
    }
    __syncthreads();
    if (tid < MV_ROWS && r_base + tid < n_out) out[(size_t)pair * n_out + r_base + tid] = red[0][tid] + red[1][tid];
}

// ---- many pairs of one matrix -----------------------------------------------------------
// grid (ceil(n_out / 64), ceil(pairs / 32)); the same warp layout.  The digits of 32 pairs are staged 512 k at a time.  Making
// them was half of the instructions, so the CS blocks of a cluster, row blocks of the same pairs, make a share each and store
// it to all of them through distributed shared memory (512 pairs: [1024 x 3072] Q4_K 79 -> 68 us,
// [3072 x 1024] Q6_K 114 -> 108).
constexpr int MM_COLS = 32, MM_KC = 512;
// bytes of a pair's digits: the columns of one load instruction (8 bytes a lane for Q4_K, 4 for Q6_K) cover distinct banks
template <int DT>
constexpr int MM_PITCH = MV_NDIG * MM_KC + (DT == LMOE_Q4_K ? 32 : 16);
template <int DT, int CS>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(MV_THREADS, 2)
mv_multi_kernel(const uint8_t *__restrict__ w, int n_out, int k, const float *__restrict__ x, int x_per_row,
                const uint32_t *__restrict__ ids, int top_k, int pairs, float *__restrict__ out) {
    pdl_begin();
    constexpr int SUB = DT == LMOE_Q4_K ? 32 : 16, NS = QK_K / SUB, BC = MM_KC / QK_K;
    constexpr int TS = DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES;
    constexpr int SP = BC * NS + 8; // f16 sums of a pair and part, padded
    extern __shared__ __align__(16) uint8_t mv_smem[];
    int8_t *xc = reinterpret_cast<int8_t *>(mv_smem);                                                    // [pair][digit][k]
    __half *sh = reinterpret_cast<__half *>(mv_smem + MM_COLS * MM_PITCH<DT>);                           // [part][pair][SP]
    float *sxs = reinterpret_cast<float *>(mv_smem + MM_COLS * MM_PITCH<DT> + MV_PARTS * MM_COLS * SP * 2); // [block][pair]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int p0 = blockIdx.y * MM_COLS, np = min(MM_COLS, pairs - p0), nb = k / QK_K;
    const int64_t row_bytes = (int64_t)nb * TS;
    const int r_base = blockIdx.x * MV_ROWS, rt = warp & 3, ks = warp >> 2;
    const int rg = min(r_base + 16 * rt + g, n_out - 1), rG = min(r_base + 16 * rt + g + 8, n_out - 1);
    const uint8_t *pg = w + (size_t)rg * row_bytes, *pG = w + (size_t)rG * row_bytes;
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    const int rank = CS > 1 ? (int)cl.block_rank() : 0;
    auto sync_all = [&]() {
        if (CS > 1) cl.sync();
        else __syncthreads();
    };
    float acc[MM_COLS / 8][4];
#pragma unroll
    for (int c = 0; c < MM_COLS / 8; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[c][i] = 0.f;
    for (int b0 = 0; b0 < nb; b0 += BC) {
        const int bn = min(BC, nb - b0);
        typename MvRaw<DT>::T raw;
        if (ks < bn) raw.load(pg + (size_t)(b0 + ks) * TS, pG + (size_t)(b0 + ks) * TS, t);
        sync_all(); // the previous chunk's digits have been read
        for (int i = rank * (MV_THREADS / 32) + warp; i < np * bn; i += CS * (MV_THREADS / 32)) {
            const int p = i / bn, b = i - p * bn, pair = p0 + p;
            MvX in;
            in.load(x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k + (size_t)(b0 + b) * QK_K,
                    ids == nullptr || ids[pair] == 0u, lane);
            uint2 dig[MV_NDIG];
            float sx;
            __half part[MV_PARTS];
            mv_digits<SUB>(in, dig, sx, part);
#pragma unroll
            for (int r = 0; r < CS; r++) {
                int8_t *xr = CS > 1 ? cl.map_shared_rank(xc, r) : xc;
                __half *hr = CS > 1 ? cl.map_shared_rank(sh, r) : sh;
                float *fr = CS > 1 ? cl.map_shared_rank(sxs, r) : sxs;
#pragma unroll
                for (int d = 0; d < MV_NDIG; d++) *reinterpret_cast<uint2 *>(xr + p * MM_PITCH<DT> + d * MM_KC + b * QK_K + lane * 8) = dig[d];
                if ((lane & (SUB / 8 - 1)) == 0) {
#pragma unroll
                    for (int h = 0; h < MV_PARTS; h++) hr[(h * MM_COLS + p) * SP + b * NS + lane / (SUB / 8)] = part[h];
                }
                if (lane == 0) fr[b * MM_COLS + p] = sx;
            }
        }
        sync_all();
        static_assert(BC == 2, "a block for each half");
        if (const int b = ks; b < bn) {
            MvA<DT> A;
            A.unpack(raw, t);
#pragma unroll
            for (int c = 0; c < MM_COLS / 8; c++) {
                if (8 * c < np) { // columns past the last pair hold whatever was there: their results are not written
                    const int8_t *xp = xc + (8 * c + g) * MM_PITCH<DT> + b * QK_K;
                    // digits from the least significant on, so that only the last addition rounds at the size of the sum.  The
                    // Q6_K offset comes off digit by digit: both terms are exact, and larger than their difference.
                    float sum[4] = {0.f, 0.f, 0.f, 0.f}, tot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int d = MV_NDIG - 1; d >= 0; d--) {
                        int al[4] = {0, 0, 0, 0};
#pragma unroll
                        for (int i = 0; i < MvA<DT>::N; i++) {
                            int f[4];
                            A.mma(i, f, xp + d * MM_KC, t);
                            const int sg = A.sg(i), sG = A.sG(i);
                            al[0] += sg * f[0]; al[1] += sg * f[1]; al[2] += sG * f[2]; al[3] += sG * f[3];
                        }
                        float cm[4] = {0.f, 0.f, 0.f, 0.f};
                        if (d < MV_PARTS) {
                            const __half *sp = sh + (d * MM_COLS + 8 * c + g) * SP + b * NS + 2 * t;
                            mma16816_acc(cm, A.f, *reinterpret_cast<const uint32_t *>(sp), NS == 16 ? *reinterpret_cast<const uint32_t *>(sp + 8) : 0u);
                        }
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (DT == LMOE_Q6_K) tot[i] += __fmaf_rn(mv_digit_weight(d), (float)al[i], -MV_OFFSET * cm[i]);
                            else tot[i] += mv_digit_weight(d) * (float)al[i], sum[i] += cm[i];
                        }
                    }
                    const float2 sx = *reinterpret_cast<const float2 *>(sxs + b * MM_COLS + 8 * c + 2 * t);
                    acc[c][0] += sx.x * (A.dg * tot[0] - A.mg * sum[0]);
                    acc[c][1] += sx.y * (A.dg * tot[1] - A.mg * sum[1]);
                    acc[c][2] += sx.x * (A.dG * tot[2] - A.mG * sum[2]);
                    acc[c][3] += sx.y * (A.dG * tot[3] - A.mG * sum[3]);
                }
            }
        }
    }
    // the two K halves meet in shared memory ([pair][row], the digits are no longer needed), then whole rows leave
    __syncthreads();
    float *red = reinterpret_cast<float *>(mv_smem);
    for (int h = 0; h < 2; h++) {
        if (ks == h) {
#pragma unroll
            for (int c = 0; c < MM_COLS / 8; c++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float *r = red + (8 * c + 2 * t + (i & 1)) * (MV_ROWS + 1) + 16 * rt + g + 8 * (i >> 1);
                    *r = h ? *r + acc[c][i] : acc[c][i];
                }
        }
        __syncthreads();
    }
    for (int i = tid; i < np * MV_ROWS; i += MV_THREADS) {
        const int p = i / MV_ROWS, r = i - p * MV_ROWS;
        // an id other than 0 names no matrix of this stack: a zero row
        if (r_base + r < n_out) out[(size_t)(p0 + p) * n_out + r_base + r] = red[p * (MV_ROWS + 1) + r];
    }
}

// ---- pairs grouped by expert ------------------------------------------------------------
// grid (row splits, pairs): a block serves one expert's next 2 * NT pairs (its "leader" is the first of them; the blocks of
// the others leave at once) on a range of row units.  A unit is 16 * m whole rows, contiguous in memory: a producer warp keeps
// a ring of units filled with one bulk copy each, NG groups of four warps take them in turn and split a unit over K (and
// over its row tiles when a row has fewer than four super-blocks).  Two pairs share one MMA (four columns each: their
// digits), so a super-block is unpacked once for 2 * NT pairs;
// four pairs a block measured no better than two where the weights of the second pass come from the L2 cache.
constexpr int MX_GW = 4;                                    // warps of a group
constexpr int MX_STAGES = 8;                                // most ring stages
constexpr int MX_WINDOW = 2048;                             // pairs of one expert are looked for among this many
constexpr int MX_UNIT = 28 * 1024;                          // a unit has as many row tiles as fit here (at least what the warps need)
constexpr int64_t MX_L2 = 100 << 20;                          // what of the 126 MB L2 cache a matrix may hope for
constexpr int MX_SMEM_ONE = 227 * 1024 - 128, MX_SMEM_TWO = 112 * 1024; // dynamic shared memory of one / two blocks a SM

struct MxLayout {
    int pitch, ns, kw, m, unit_bytes, stride, nstage, o_sum, o_sx, o_red, o_bar, o_ring, total;
    __host__ __device__ MxLayout(bool q4, int np, int ng, int nb, int smem_max) {
        const int row_bytes = nb * (q4 ? Q4K_BYTES : Q6K_BYTES);
        ns = q4 ? 8 : 16;
        pitch = nb * QK_K + (q4 ? 32 : 16); // the columns of one load instruction cover distinct banks
        kw = nb >= 4 ? 4 : (nb >= 2 ? 2 : 1); // warps along K; 4 / kw along the row tiles
        m = 4 / kw;
        while (2 * m * kw <= 8 && 32 * m * row_bytes <= MX_UNIT) m *= 2;
        unit_bytes = 16 * m * row_bytes;
        stride = (unit_bytes + (q4 ? 0 : 16) + 127) / 128 * 128; // Q6_K: an aligned two-word read may end past the last block
        int o = np * MV_NDIG * pitch;
        o_sum = o; o += np * MV_PARTS * nb * ns * 2;
        o_sx = o; o += (np * nb * 4 + 15) / 16 * 16;
        o_red = o; o += ng * 2 * kw * np * 16 * m * 4;
        o_bar = o; o += 2 * MX_STAGES * 8 + 16;
        o_ring = (o + 127) / 128 * 128;
        nstage = (smem_max - o_ring) / stride;
        nstage = nstage > MX_STAGES ? MX_STAGES : (nstage < 0 ? 0 : nstage);
        total = o_ring + nstage * stride;
    }
};

// One super-block of two rows against the digits of 2 * NT pairs.  y[j]: this lane's pair of column tile j, rows g and G;
// lanes of even t hold the two high digits and parts of the sums, lanes of odd t the low ones (no part in the last column).
template <int DT, int NT>
__device__ __forceinline__ void mx_finish(const int (&al)[NT][4], const float (&cm)[NT][4], float dg, float dG, float mg, float mG, int b, int t,
                                          const float *const (&sxp)[NT], float (&y)[NT][2]) {
    const float f0 = (t & 1) ? 256.f : 16777216.f, f1 = (t & 1) ? 1.f : 65536.f, m1 = (t & 1) ? 0.f : 1.f;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const float sx = sxp[j][b];
        if (DT == LMOE_Q6_K) { // the offset comes off digit by digit: both terms are exact, and larger than their difference
            const float k1 = m1 * -MV_OFFSET;
            y[j][0] += sx * dg * (__fmaf_rn(f0, (float)al[j][0], -MV_OFFSET * cm[j][0]) + __fmaf_rn(f1, (float)al[j][1], k1 * cm[j][1]));
            y[j][1] += sx * dG * (__fmaf_rn(f0, (float)al[j][2], -MV_OFFSET * cm[j][2]) + __fmaf_rn(f1, (float)al[j][3], k1 * cm[j][3]));
        } else {
            y[j][0] += sx * (dg * (f0 * (float)al[j][0] + f1 * (float)al[j][1]) - mg * (cm[j][0] + m1 * cm[j][1]));
            y[j][1] += sx * (dG * (f0 * (float)al[j][2] + f1 * (float)al[j][3]) - mG * (cm[j][2] + m1 * cm[j][3]));
        }
    }
}
template <int NT>
__device__ __forceinline__ void mx_q4k(const uint8_t *bg, const uint8_t *bG, int b, int t, const int8_t *const (&xcol)[NT],
                                       const __half *const (&scol)[NT], const float *const (&sxp)[NT], float (&y)[NT][2]) {
    MvQ4 R;
    R.hg = *reinterpret_cast<const uint4 *>(bg);
    R.hG = *reinterpret_cast<const uint4 *>(bG);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        R.wg[j] = *reinterpret_cast<const uint2 *>(bg + 16 + 32 * j + 8 * t);
        R.wG[j] = *reinterpret_cast<const uint2 *>(bG + 16 + 32 * j + 8 * t);
    }
    MvA<LMOE_Q4_K> A;
    A.unpack(R, t);
    int al[NT][4];
    float cm[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        mma16816_z(cm[j], A.f[0], A.f[1], 0u, 0u, *reinterpret_cast<const uint32_t *>(scol[j] + b * 8 + 2 * t), 0u);
#pragma unroll
        for (int q = 0; q < 4; q++) al[j][q] = 0;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int sg = A.sg(i), sG = A.sG(i);
#pragma unroll
        for (int j = 0; j < NT; j++) {
            int f[4];
            A.mma(i, f, xcol[j] + b * QK_K, t);
            al[j][0] += sg * f[0]; al[j][1] += sg * f[1]; al[j][2] += sG * f[2]; al[j][3] += sG * f[3];
        }
    }
    mx_finish<LMOE_Q4_K, NT>(al, cm, A.dg, A.dG, A.mg, A.mG, b, t, sxp, y);
}
template <int NT, int MIS>
__device__ __forceinline__ void mx_q6k(const uint8_t *bg, const uint8_t *bG, int b, int t, const int8_t *const (&xcol)[NT],
                                       const __half *const (&scol)[NT], const float *const (&sxp)[NT], float (&y)[NT][2]) {
    constexpr uint32_t M4 = 0x0F0F0F0Fu, M2 = 0x30303030u;
    const int8_t *cg = reinterpret_cast<const int8_t *>(bg + 192), *cG = reinterpret_cast<const int8_t *>(bG + 192);
    const float dg = lmoe_h2f(*reinterpret_cast<const uint16_t *>(bg + 208)), dG = lmoe_h2f(*reinterpret_cast<const uint16_t *>(bG + 208));
    int al[NT][4];
    float cm[NT][4];
    {
        const uint32_t f0 = sc_pair_half2(cg + 2 * t), f1 = sc_pair_half2(cG + 2 * t), f2 = sc_pair_half2(cg + 2 * t + 8), f3 = sc_pair_half2(cG + 2 * t + 8);
#pragma unroll
        for (int j = 0; j < NT; j++) {
            mma16816_z(cm[j], f0, f1, f2, f3, *reinterpret_cast<const uint32_t *>(scol[j] + b * 16 + 2 * t),
                       *reinterpret_cast<const uint32_t *>(scol[j] + b * 16 + 2 * t + 8));
#pragma unroll
            for (int q = 0; q < 4; q++) al[j][q] = 0;
        }
    }
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const uint32_t wg0 = lds32<MIS>(bg, 192 + 8 * n), wg1 = lds32<MIS>(bg, 196 + 8 * n);
        const uint32_t wG0 = lds32<MIS>(bG, 192 + 8 * n), wG1 = lds32<MIS>(bG, 196 + 8 * n);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int l0 = 16 * c + 4 * t;
            const uint32_t qa_g = lds32<MIS>(bg, 64 * n + l0), qb_g = lds32<MIS>(bg, 64 * n + 32 + l0), qh_g = lds32<MIS>(bg, 128 + 32 * n + l0);
            const uint32_t qa_G = lds32<MIS>(bG, 64 * n + l0), qb_G = lds32<MIS>(bG, 64 * n + 32 + l0), qh_G = lds32<MIS>(bG, 128 + 32 * n + l0);
#pragma unroll
            for (int i = 0; i < 4; i++) { // sub-block 8 n + 2 i + c: nibble i / 2 of ql run 2 (i & 1) + c, bits 2 i of qh run c
                const uint32_t qg = (i & 1) ? qb_g : qa_g, qG = (i & 1) ? qb_G : qa_G;
                const uint32_t lg = (i & 2) ? (qg >> 4) : qg, lG = (i & 2) ? (qG >> 4) : qG;
                const uint32_t hg = i == 0 ? (qh_g << 4) : (i == 1 ? (qh_g << 2) : (i == 2 ? qh_g : (qh_g >> 2)));
                const uint32_t hG = i == 0 ? (qh_G << 4) : (i == 1 ? (qh_G << 2) : (i == 2 ? qh_G : (qh_G >> 2)));
                const uint32_t a0 = (lg & M4) | (hg & M2), a1 = (lG & M4) | (hG & M2);
                const int sg = sbyte(i < 2 ? wg0 : wg1, 2 * (i & 1) + c), sG = sbyte(i < 2 ? wG0 : wG1, 2 * (i & 1) + c);
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    int f[4];
                    imma16816_z(f, a0, a1, *reinterpret_cast<const uint32_t *>(xcol[j] + b * QK_K + 128 * n + 32 * i + l0));
                    al[j][0] += sg * f[0]; al[j][1] += sg * f[1]; al[j][2] += sG * f[2]; al[j][3] += sG * f[3];
                }
            }
        }
    }
    mx_finish<LMOE_Q6_K, NT>(al, cm, dg, dG, 0.f, 0.f, b, t, sxp, y);
}

struct MxArgs {
    const uint8_t *w; // the expert's rows
    const uint8_t *ring;
    const int8_t *xc;
    const __half *sums;
    const float *sxs;
    float *red, *out;
    uint64_t *full, *empty;
    uint32_t *fail; // the block's failure words, then the count of units issued
    const int *pairs;
    int np, n_out, nb, u0, u1;
};

// The units of a block, by the consumer warps: columns of NT MMA tiles.
template <int DT, int NT, int NG>
__device__ __forceinline__ void mx_units(const MxArgs P, const MxLayout L, int warp_all, int lane) {
    const int gi = warp_all / MX_GW, wq = warp_all % MX_GW, g = lane >> 2, t = lane & 3;
    const int kq = wq % L.kw, tq = wq / L.kw, tstep = MX_GW / L.kw;
    constexpr int TS = DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES;
    const int nb = P.nb, row_bytes = nb * TS, rows = 16 * L.m;
    const int8_t *xcol[NT];
    const __half *scol[NT];
    const float *sxp[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int pb = 2 * j + (g >> 2), po = 2 * j + (t >> 1); // pair of this lane's B column, and of its accumulators
        xcol[j] = P.xc + ((pb < P.np ? pb : 0) * MV_NDIG + (g & 3)) * L.pitch;
        scol[j] = P.sums + ((pb < P.np ? pb : 0) * MV_PARTS + min(g & 3, MV_PARTS - 1)) * nb * L.ns;
        sxp[j] = P.sxs + (po < P.np ? po : 0) * nb;
    }
    // Q6_K rows 2g and 2g + 1 where they are word aligned: the eight rows of a load sit in disjoint banks
    const bool inter = DT == LMOE_Q6_K && (row_bytes & 2) == 0;
    const int rowA = inter ? 2 * g : g, rowB = inter ? 2 * g + 1 : g + 8;
    int seq = gi; // of the block's unit sequence
    for (int u = P.u0 + gi; u < P.u1; u += NG, seq += NG) {
        const int s = seq % L.nstage;
        wait_issued(P.fail + 3, (uint32_t)seq, P.fail, 1u);
        mbar_wait(P.full + s, (uint32_t)((seq / L.nstage) & 1), P.fail, 1u);
        float *rb = P.red + (gi * 2 + ((seq / NG) & 1)) * L.kw * 2 * NT * rows;
        for (int tile = tq; tile < L.m; tile += tstep) {
            const uint8_t *rg = P.ring + (size_t)s * L.stride + (16 * tile + rowA) * row_bytes;
            const uint8_t *rG = P.ring + (size_t)s * L.stride + (16 * tile + rowB) * row_bytes;
            float y[NT][2];
#pragma unroll
            for (int j = 0; j < NT; j++) y[j][0] = y[j][1] = 0.f;
            for (int b = kq; b < nb; b += L.kw) {
                if (DT == LMOE_Q4_K) mx_q4k<NT>(rg + b * TS, rG + b * TS, b, t, xcol, scol, sxp, y);
                else if (row_bytes & 2) mx_q6k<NT, 2>(rg + b * TS, rG + b * TS, b, t, xcol, scol, sxp, y);
                else if (b & 1) mx_q6k<NT, 1>(rg + b * TS, rG + b * TS, b, t, xcol, scol, sxp, y);
                else mx_q6k<NT, 0>(rg + b * TS, rG + b * TS, b, t, xcol, scol, sxp, y);
            }
#pragma unroll
            for (int j = 0; j < NT; j++) {
                y[j][0] += __shfl_xor_sync(0xffffffffu, y[j][0], 1);
                y[j][1] += __shfl_xor_sync(0xffffffffu, y[j][1], 1);
                if ((t & 1) == 0) {
                    float *r = rb + (kq * 2 * NT + 2 * j + (t >> 1)) * rows + 16 * tile;
                    r[rowA] = y[j][0];
                    r[rowB] = y[j][1];
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(P.empty + s);
        // the buffer is written again two units of the group later, after the group's next barrier, which a warp reaches
        // only when it has read this one
        bar_sync(2 + gi, 32 * MX_GW);
        const int r0 = u * rows, nr = min(rows, P.n_out - r0);
        for (int i = wq * 32 + lane; i < P.np * rows; i += 32 * MX_GW) {
            const int p = i / rows, r = i - p * rows;
            float sum = 0.f;
            for (int q = 0; q < L.kw; q++) sum += rb[(q * 2 * NT + p) * rows + r];
            if (*reinterpret_cast<volatile uint32_t *>(P.fail) != 0u) sum = __int_as_float(0x7fc00000);
            if (r < nr) P.out[(size_t)P.pairs[p] * P.n_out + r0 + r] = sum;
        }
    }
}

// N = MV_JOBS: up to as many products of the same shape in one launch, blockIdx.z each (see launch_mul_mv_id_jobs).  N = 1: one, its
// job at a place known to the compiler (Q6_K [4096 x 1024], 16 pairs: 14.5 us, with the job behind blockIdx.z 15.5).
template <int N>
struct MxJobs {
    MvJob job[N];
};
template <int DT, int NT, int NG, bool ODD, int N>
__global__ void __launch_bounds__(32 * (NG * MX_GW + 1), NG == 2 ? 2 : 1)
mv_expert_kernel(const __grid_constant__ MxJobs<N> jobs, int n_out, int k, int smem_max) {
    pdl_begin();
    const MvJob &J = jobs.job[N == 1 ? 0 : blockIdx.z];
    const uint8_t *__restrict__ w = J.w;
    const int64_t expert_bytes = J.expert_bytes;
    const float *__restrict__ x = J.x;
    const uint32_t *__restrict__ ids = J.ids;
    float *__restrict__ out = J.out;
    const int n_expert = J.n_expert, x_per_row = J.x_per_row, top_k = J.top_k, n_pairs = J.pairs;
    if (N > 1 && (int)blockIdx.y >= n_pairs) return;
    constexpr int SUB = DT == LMOE_Q4_K ? 32 : 16, NS = QK_K / SUB, NP = 2 * NT, CONS_WARPS = NG * MX_GW;
    extern __shared__ __align__(128) uint8_t mx_smem[];
    __shared__ int pairs_s[NP], np_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, p0 = blockIdx.y;
    const int nb = k / QK_K;
    const MxLayout L(DT == LMOE_Q4_K, NP, NG, nb, smem_max);
    const int rows = 16 * L.m, units = (n_out + rows - 1) / rows;
    const int u0 = (int)((int64_t)units * blockIdx.x / gridDim.x), u1 = (int)((int64_t)units * (blockIdx.x + 1) / gridDim.x);
    const uint32_t e = ids ? __ldg(ids + p0) : 0u;
    if (e >= (uint32_t)n_expert) { // an out-of-range id produces a zero row
        for (int i = u0 * rows + tid; i < min(u1 * rows, n_out); i += 32 * (CONS_WARPS + 1)) out[(size_t)p0 * n_out + i] = 0.f;
        return;
    }
    uint64_t *full = reinterpret_cast<uint64_t *>(mx_smem + L.o_bar), *empty = full + MX_STAGES;
    uint32_t *fail = reinterpret_cast<uint32_t *>(empty + MX_STAGES);
    if (warp == 0) { // the expert's pairs: a count of those before p0 in the window, a list from p0 on
        const int w0 = p0 / MX_WINDOW * MX_WINDOW, w1 = min(w0 + MX_WINDOW, n_pairs);
        int before = 0, found = 0;
        for (int i0 = w0; i0 < w1 && found < NP; i0 += 256) {
            uint32_t id[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int i = i0 + 32 * j + lane;
                id[j] = i < w1 ? (ids ? __ldg(ids + i) : 0u) : 0xffffffffu;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int i = i0 + 32 * j + lane;
                const uint32_t hit = __ballot_sync(0xffffffffu, id[j] == e && i < w1), old = __ballot_sync(0xffffffffu, i < p0);
                before += __popc(hit & old);
                const uint32_t now = hit & ~old;
                const int pos = found + __popc(now & ((1u << lane) - 1u));
                if (((now >> lane) & 1u) && pos < NP) pairs_s[pos] = i;
                found += __popc(now);
            }
            if (i0 + 256 > p0 && (before & (NP - 1))) break;
        }
        if (lane == 0) np_s = (before & (NP - 1)) ? 0 : min(found, NP);
    } else if (tid == 32) {
        for (int s = 0; s < L.nstage; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, MX_GW);
        }
        fail[0] = fail[1] = fail[2] = fail[3] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int np = np_s;
    if (np == 0) return; // an earlier pair's block serves this one
    const uint8_t *we = w + (size_t)e * expert_bytes;
    if (warp == CONS_WARPS) {
        if (lane == 0) {
            const int64_t row_bytes = (int64_t)nb * (DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES);
            int i = 0;
            for (int u = u0; u < u1; u++, i++) {
                const int s = i % L.nstage;
                if (i >= L.nstage) mbar_wait<32>(empty + s, (uint32_t)((i / L.nstage - 1) & 1), fail, 2u);
                copy_rows<ODD>(mx_smem + L.o_ring + (size_t)s * L.stride, we + (size_t)u * L.unit_bytes, (uint32_t)(min(rows, n_out - u * rows) * row_bytes), full + s);
                set_issued(fail + 3, (uint32_t)i + 1);
            }
            // leave only when the last copies have landed (they have been waited for already unless a consumer gave up)
            for (int j = i > L.nstage ? i - L.nstage : 0; j < i; j++)
                mbar_wait<32>(full + j % L.nstage, (uint32_t)((j / L.nstage) & 1), fail, 3u);
        }
        return;
    }
    int8_t *xc = reinterpret_cast<int8_t *>(mx_smem);
    __half *sums = reinterpret_cast<__half *>(mx_smem + L.o_sum);
    float *sxs = reinterpret_cast<float *>(mx_smem + L.o_sx);
    auto src = [&](int i) {
        const int pair = pairs_s[i / nb];
        return x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k + (size_t)(i % nb) * QK_K;
    };
    MvX in;
    if (warp < np * nb) in.load(src(warp), true, lane);
    for (int i = warp; i < np * nb; i += CONS_WARPS) {
        const int p = i / nb, b = i - p * nb;
        MvX next;
        if (i + CONS_WARPS < np * nb) next.load(src(i + CONS_WARPS), true, lane);
        uint2 dig[MV_NDIG];
        float sx;
        __half part[MV_PARTS];
        mv_digits<SUB>(in, dig, sx, part);
        in = next;
#pragma unroll
        for (int d = 0; d < MV_NDIG; d++) *reinterpret_cast<uint2 *>(xc + (p * MV_NDIG + d) * L.pitch + b * QK_K + lane * 8) = dig[d];
        if ((lane & (SUB / 8 - 1)) == 0) {
#pragma unroll
            for (int h = 0; h < MV_PARTS; h++) sums[((MV_PARTS * p + h) * nb + b) * NS + lane / (SUB / 8)] = part[h];
        }
        if (lane == 0) sxs[p * nb + b] = sx;
    }
    bar_sync(1, 32 * CONS_WARPS);
    const MxArgs P = {we, mx_smem + L.o_ring, xc, sums, sxs, reinterpret_cast<float *>(mx_smem + L.o_red), out, full, empty, fail, pairs_s,
                      np, n_out, nb, u0, u1};
    mx_units<DT, NT, NG>(P, L, warp, lane);
}

template <int DT, int NT, int NG, bool ODD, int N>
cudaError_t launch_mv_expert_jobs(const MvJob *job, int jobs, int n_out, int k, int dev, int sms, cudaStream_t s) {
    constexpr int smem_max = NG == 2 ? MX_SMEM_TWO : MX_SMEM_ONE;
    if (k > smem_max) return cudaErrorNotSupported; // the digits alone are longer, and the layout's sums stay within 32 bits
    const MxLayout L(DT == LMOE_Q4_K, 2 * NT, NG, k / QK_K, smem_max);
    if (L.nstage < NG) return cudaErrorNotSupported; // rows too long for the ring
    static thread_local int c_dev = -1;
    if (dev != c_dev) {
        const cudaError_t e = cudaFuncSetAttribute(mv_expert_kernel<DT, NT, NG, ODD, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e != cudaSuccess) return e;
        c_dev = dev;
    }
    const int64_t units = (n_out + 16 * L.m - 1) / (16 * L.m), slots = (NG == 2 ? 2 : 1) * (int64_t)sms;
    // Row splits: the blocks run in rounds of `slots`, and a block costs about three units of start-up.
    MxJobs<N> P = {};
    int64_t groups = 0, most = 0;
    for (int j = 0; j < jobs; j++) {
        P.job[j] = job[j];
        groups += job[j].n_expert == 1 ? (job[j].pairs + 2 * NT - 1) / (2 * NT) : job[j].pairs;
        most = job[j].pairs > most ? job[j].pairs : most;
    }
    int64_t gx = 1, best = INT64_MAX;
    for (int64_t rounds = 1; rounds <= 16; rounds++) {
        int64_t g = rounds * slots / groups;
        g = g < 1 ? 1 : (g > units ? units : g);
        const int64_t cost = (groups * g + slots - 1) / slots * (3 + (units + g - 1) / g);
        if (cost < best) best = cost, gx = g;
    }
    launch_pdl(mv_expert_kernel<DT, NT, NG, ODD, N>, dim3((unsigned)gx, (unsigned)most, (unsigned)jobs), 32 * (NG * MX_GW + 1), L.total, s, P, n_out, k,
               smem_max);
    return cudaGetLastError();
}

template <int DT, int NT, int NG, bool ODD>
cudaError_t launch_mv_expert(const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *x, int64_t pairs, int x_per_row,
                             const uint32_t *ids, int top_k, float *out, int dev, int sms, cudaStream_t s) {
    const int64_t step = 65535 / top_k * top_k; // grid.y is limited to 65535
    for (int64_t p = 0; p < pairs; p += step) {
        const MvJob job = {w, expert_bytes, n_expert, x + (size_t)(p / top_k) * x_per_row * k, x_per_row, ids ? ids + p : nullptr, top_k,
                           (int)(pairs - p < step ? pairs - p : step), out + (size_t)p * n_out};
        const cudaError_t r = launch_mv_expert_jobs<DT, NT, NG, ODD, 1>(&job, 1, n_out, k, dev, sms, s);
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

// One block an SM, with twice the warps on the same digits: where a row is too long for two, and for a single matrix that is
// larger than the L2 cache, so that up to four pairs cost one pass over it ([100352 x 3072] Q6_K, 2 / 4 pairs: 86 / 172 us in
// passes of one pair, 52 / 72 so; with three digits a value 47 / 72, and 55 / 91 with two blocks an SM).
template <int DT, bool ODD>
cudaError_t launch_mv_by_expert(const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *x, int64_t pairs,
                                int x_per_row, const uint32_t *ids, int top_k, float *out, int dev, int sms, cudaStream_t s) {
    cudaError_t r = cudaErrorNotSupported;
    if (n_expert == 1 && expert_bytes > MX_L2)
        r = pairs > 2 ? launch_mv_expert<DT, 2, 4, ODD>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s)
                      : launch_mv_expert<DT, 1, 4, ODD>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s);
    if (r == cudaErrorNotSupported) r = launch_mv_expert<DT, 1, 2, ODD>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s);
    if (r == cudaErrorNotSupported) r = launch_mv_expert<DT, 1, 4, ODD>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s);
    return r;
}

// Where the warp-per-row kernel is the faster one.  The others begin with 2 us of setting up digits, ring and barriers, which
// pays from a number of rows (pairs times rows of the matrix) on that falls with a row's length, and they work on 16 rows or
// more at a time.  Row kernel against the others: Q4_K [1024 x 512], 4 / 8 pairs 3.7 / 5.0 us against 4.2 / 4.3,
// [1024 x 3072], 1 / 4 pairs 5.0 / 9.7 against 5.2 / 7.3, [7 x 512], 1024 pairs 4.7 against 14.4; Q6_K [1024 x 1024],
// 4 / 16 pairs 4.3 / 9.6 against 5.2 / 8.6, [256 x 2048], 1 / 64 pairs 5.4 / 15.6 against 5.0 / 13.4.
template <int DT>
bool mv_rows_better(int64_t pairs, int n_out, int k) {
    const int64_t rows = pairs * n_out;
    if (DT == LMOE_Q4_K)
        return rows < (k < 1024 ? 8192 : (k < 2048 ? 4096 : (k < 3072 ? 2560 : 2048))) || n_out < (k < 2048 ? 32 : 16);
    return k < 2048 ? rows < (k < 1024 ? 16384 : 8193) || n_out < 64 : n_out < 32;
}

template <int DT>
cudaError_t launch_mv_rows(const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *x, int64_t pairs, int x_per_row,
                           const uint32_t *ids, int top_k, float *out, cudaStream_t s) {
    const int64_t step = 65535 / top_k * top_k; // grid.y is limited to 65535
    for (int64_t p = 0; p < pairs; p += step) {
        const int64_t n = pairs - p < step ? pairs - p : step;
        // launched the plain way: blocks that move in beside the previous kernel are spread unevenly over the SMs (64 rows of 32768
        // Q6_K, 128 pairs: 157 us overlapped, 106 plain)
        mv_row_kernel<DT><<<dim3((unsigned)((n_out + MR_WARPS * MR_ROWS - 1) / (MR_WARPS * MR_ROWS)), (unsigned)n), MR_WARPS * 32, 0, s>>>(
            w, expert_bytes, n_expert, n_out, k, x + (size_t)(p / top_k) * x_per_row * k, x_per_row, ids ? ids + p : nullptr, top_k,
            out + (size_t)p * n_out);
    }
    return cudaGetLastError();
}

cudaError_t mv_device(int &dev, int &sms) {
    cudaError_t e = cudaGetDevice(&dev);
    static thread_local int c_dev = -1, c_sms = 0;
    if (e == cudaSuccess && dev != c_dev && (e = cudaDeviceGetAttribute(&c_sms, cudaDevAttrMultiProcessorCount, dev)) == cudaSuccess) c_dev = dev;
    sms = c_sms;
    return e;
}
bool mv_multi_better(int n_expert, int n_out, int64_t pairs, int sms) {
    return n_expert == 1 && (pairs + MM_COLS - 1) / MM_COLS * ((n_out + MV_ROWS - 1) / MV_ROWS) >= sms && pairs > 4;
}
// The tensor-core kernel of mv_dense.cu takes a super-block of 128 rows and 32 pairs at a time, 3.7 us Q4_K, 4.9 Q6_K, whatever the number
// of blocks on the device; these kernels' time goes with the work.  us here / there, cold L2:
//   pairs                      32           64          128          256          512         1024         4096
//   [1024 x 3072] Q4_K  21.5 / 48.1  31.8 / 49.2  34.8 / 49.2  55.5 / 49.2  71.7 / 49.3   137 / 94.2    473 / 309
//   [768 x 2048] Q4_K   18.5 / 36.9  22.6 / 36.9  27.6 / 36.9  42.0 / 36.9  49.2 / 37.1  76.8 / 69.6    244 / 195
//   [3072 x 1024] Q6_K  23.5 / 24.6  41.0 / 24.6  43.0 / 25.6  67.6 / 45.1   115 / 65.5   206 / 122     787 / 410
//   [2048 x 768] Q6_K   22.6 / 20.6  34.8 / 20.7  45.1 / 20.5  37.9 / 22.5  69.6 / 36.9   129 / 68.7    442 / 224
// Of 264 matrices and counts that the rule sends there, drawn from 5 to 100352 rows of 256 to 12288 and 64 to 16384 pairs, one is longer there
// ([768 x 2048] Q6_K, 160 pairs: 38.9 / 41.0), the rest take 0.2 to 1.0 times as long.
// Below 64 pairs a chain's shared product is better off in the launch of the routed ones (48 tokens op by op, 256 experts: 443 us so, 460 apart).
bool mv_dense_better(int dt, const uint8_t *w, int n_expert, int n_out, int k, int64_t pairs, int sms) {
    if (n_expert != 1 || pairs < 64 || (reinterpret_cast<uintptr_t>(w) & 15u)) return false;
    const bool q4 = dt == LMOE_Q4_K, multi = mv_multi_better(n_expert, n_out, pairs, sms);
    const int64_t rounds = (((int64_t)n_out + 127) / 128 * ((pairs + 31) / 32) + sms - 1) / sms;
    const double there = 5.0 + (double)rounds * (k / QK_K) * (q4 ? 3.7 : 4.9);
    return there < 7.0 + (double)pairs * n_out * k * (multi ? (q4 ? 4.2e-8 : 6.8e-8) : (q4 ? 6.0e-8 : 1.5e-7));
}
// a bulk copy starts and ends on 16 bytes: every expert must; the end of a single matrix may be ragged
bool mv_copies(const uint8_t *w, int n_expert, int64_t expert_bytes) {
    return (reinterpret_cast<uintptr_t>(w) & 15u) == 0 && (n_expert == 1 || expert_bytes % 16 == 0);
}

template <int DT>
cudaError_t launch_mv(const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *x, int64_t pairs, int x_per_row,
                      const uint32_t *ids, int top_k, float *out, cudaStream_t s) {
    if (mv_rows_better<DT>(pairs, n_out, k)) return launch_mv_rows<DT>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, s);
    constexpr int NS = DT == LMOE_Q4_K ? 8 : 16;
    const unsigned gx = (unsigned)((n_out + MV_ROWS - 1) / MV_ROWS);
    int dev, sms;
    cudaError_t e = mv_device(dev, sms);
    if (e != cudaSuccess) return e;
    if (mv_dense_better(DT, w, n_expert, n_out, k, pairs, sms)) return launch_mv_dense(DT, w, n_out, k, x, pairs, x_per_row, ids, top_k, out, s);
    // One matrix for all pairs: 32 pairs to an unpacked super-block, once such blocks cover every SM.  (Below that two pairs to a
    // block win by parallelism: [1024 x 3072] Q4_K, 64 / 512 pairs 26 / 92 us against 44 / 68, [3072 x 1024] Q6_K, 32 / 128
    // pairs 19 / 44 against 26 / 39.)
    if (mv_multi_better(n_expert, n_out, pairs, sms)) {
        constexpr int smem = MM_COLS * MM_PITCH<DT> + MV_PARTS * MM_COLS * (MM_KC / QK_K * NS + 8) * 2 + (MM_KC / QK_K) * MM_COLS * 4;
        constexpr int CS = 4;
        static thread_local int c_dev = -1;
        if (dev != c_dev) {
            if ((e = cudaFuncSetAttribute(mv_multi_kernel<DT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
            if ((e = cudaFuncSetAttribute(mv_multi_kernel<DT, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
            c_dev = dev;
        }
        // clusters where the row blocks that fill up the last one are few (they only make digits)
        const bool cluster = gx % CS == 0 || gx >= 4 * CS;
        // grid.y is limited to 65535 groups
        const int64_t step = (int64_t)65535 * MM_COLS / top_k * top_k;
        for (int64_t p = 0; p < pairs; p += step) {
            const int64_t n = pairs - p < step ? pairs - p : step;
            launch_pdl(cluster ? mv_multi_kernel<DT, CS> : mv_multi_kernel<DT, 1>,
                       dim3(cluster ? (gx + CS - 1) / CS * CS : gx, (unsigned)((n + MM_COLS - 1) / MM_COLS)), MV_THREADS, smem, s, w, n_out, k,
                       x + (size_t)(p / top_k) * x_per_row * k, x_per_row, ids ? ids + p : nullptr, top_k, (int)n, out + (size_t)p * n_out);
        }
        return cudaGetLastError();
    }
    if (mv_copies(w, n_expert, expert_bytes)) {
        const cudaError_t r = expert_bytes % 16 ? launch_mv_by_expert<DT, true>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s)
                                                : launch_mv_by_expert<DT, false>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, dev, sms, s);
        if (r != cudaErrorNotSupported) return r;
    }
    // Q6_K straight from global memory takes two loads a word, which the matrix instructions do not make up for: 16 experts of
    // [256 x 8192], 64 pairs 61.2 us that way, 53.9 by rows, of [4096 x 8192], 8 pairs 125 and 107
    if (DT == LMOE_Q6_K) return launch_mv_rows<DT>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, s);
    const int bc = k / QK_K < MV_PAIR_BLOCKS ? k / QK_K : MV_PAIR_BLOCKS;
    const int smem_pair = MV_NDIG * (bc * QK_K + 32) + MV_PARTS * bc * NS * 2 + bc * 4; // at most 36 KB
    // grid.y is limited to 65535: fold large pair counts over several launches
    const int64_t step = 65535 / top_k * top_k;
    for (int64_t p = 0; p < pairs; p += step) {
        const int64_t n = pairs - p < step ? pairs - p : step;
        launch_pdl(mv_pair_kernel<LMOE_Q4_K>, dim3(gx, (unsigned)n), MV_THREADS, smem_pair, s, w, expert_bytes, n_expert, n_out, k,
                                                                                x + (size_t)(p / top_k) * x_per_row * k, x_per_row,
                                                                                ids ? ids + p : nullptr, top_k, out + (size_t)p * n_out);
    }
    return cudaGetLastError();
}

// Several products of one shape, those that mv_expert_kernel serves in one launch: a launch of it begins with 2 us of digits,
// ring and barriers on every SM and ends with the slowest block, and the products of an expert FFN that do not depend on one
// another share both.  (3 tokens op by op, ten of 256 experts [1024 x 3072] and the shared one: 112 us with twelve launches and
// eleven calls from the host, 74 with seven and two.)
template <int DT>
cudaError_t launch_mv_jobs(const MvJob *job, int jobs, int n_out, int k, cudaStream_t s) {
    int dev, sms, n = 0;
    const cudaError_t e = mv_device(dev, sms);
    if (e != cudaSuccess) return e;
    MvJob together[MV_JOBS], alone[MV_JOBS];
    int rest = 0;
    for (int j = 0; j < jobs; j++) {
        const MvJob &J = job[j];
        const bool one = J.pairs > 0 && J.pairs <= 65535 && !mv_rows_better<DT>(J.pairs, n_out, k) && !mv_multi_better(J.n_expert, n_out, J.pairs, sms) && !mv_dense_better(DT, J.w, J.n_expert, n_out, k, J.pairs, sms) &&
                         mv_copies(J.w, J.n_expert, J.expert_bytes) && J.expert_bytes % 16 == 0 && !(J.n_expert == 1 && J.expert_bytes > MX_L2);
        if (one) together[n++] = J;
        else alone[rest++] = J;
    }
    if (n > 1) {
        const cudaError_t r = launch_mv_expert_jobs<DT, 1, 2, false, MV_JOBS>(together, n, n_out, k, dev, sms, s);
        if (r == cudaSuccess) n = 0;
        else if (r != cudaErrorNotSupported) return r;
    }
    for (int j = 0; j < n + rest; j++) {
        const MvJob &J = j < n ? together[j] : alone[j - n];
        if (J.pairs == 0) continue;
        const cudaError_t r = launch_mv<DT>(J.w, J.expert_bytes, J.n_expert, n_out, k, J.x, J.pairs, J.x_per_row, J.ids, J.top_k, J.out, s);
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

} // namespace

cudaError_t launch_mul_mv_id(int dtype, const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k,
                             const float *x, int t, int x_per_row, const uint32_t *ids, int top_k, float *out,
                             cudaStream_t s) {
    if (t == 0 || top_k == 0 || n_out == 0) return cudaSuccess;
    const int64_t pairs = (int64_t)t * top_k;
    return dtype == LMOE_Q4_K ? launch_mv<LMOE_Q4_K>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, s)
                              : launch_mv<LMOE_Q6_K>(w, expert_bytes, n_expert, n_out, k, x, pairs, x_per_row, ids, top_k, out, s);
}

cudaError_t launch_mul_mv_id_jobs(int dtype, const MvJob *job, int jobs, int n_out, int k, cudaStream_t s) {
    if (jobs > MV_JOBS) return cudaErrorInvalidValue;
    if (n_out == 0) return cudaSuccess;
    return dtype == LMOE_Q4_K ? launch_mv_jobs<LMOE_Q4_K>(job, jobs, n_out, k, s) : launch_mv_jobs<LMOE_Q6_K>(job, jobs, n_out, k, s);
}
