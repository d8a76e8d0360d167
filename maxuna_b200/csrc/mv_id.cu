// Stand-alone indexed quantized mat-vec: out[t,s,:] = W[ids[t,s]] . x[t, s|0, :].
// Reference: `ops::mul_mv_id`, src/ops/mv_id.rs:37-45; kernels
// kernel_mul_mv_id_q{4,6}_K_f32_v, src/ops/mv.metal:181-290, 413-504, 638-717.
//
// Two kernels.  Both carry the activations as three signed base-256 digits under the largest magnitude of every 256-wide
// block (24 bits: the resolution of f32 at that magnitude) and multiply them with the raw 4- and 6-bit fields on the integer
// tensor-core path (mma.sync u8 x s8 -> s32, exact), as the fused decode kernel does; the scales come in once per
// super-block.  A lane-per-16-bytes f32 dot product was bound by its conversions and multiply-adds.
//   mv_pair_kernel   one (token, slot) pair per block row: the digits are MMA columns.  Weights go straight from global
//                    memory into the A fragments (a fragment row is a whole 32-byte sector).
//                    30 pairs of [1024 x 3072] Q4_K: 33 -> 20 us.
//   mv_multi_kernel  many pairs of ONE weight matrix (the shared expert, a plain matrix): eight pairs are the columns of
//                    an MMA, so a super-block is unpacked once for 32 pairs.  512 pairs of [1024 x 3072] Q4_K: 830 -> 84 us.
#include "common.cuh"
#include "stream_math.cuh"

namespace {

constexpr int MV_THREADS = 256, MV_ROWS = 64; // rows of a block: four MMA row tiles, the K dimension in two halves
constexpr int MV_NDIG = 3;
// Largest quantized magnitude: digits 127, 127, 127 is 127 * 65793; a little below, so that every digit stays in a byte.
constexpr float MV_QMAX = 8355000.f;
// The SUB-wide sums (|sum| <= 32 * QMAX < 2^28) enter an f16 product times 2^-13, as a high and a low part.
constexpr float MV_SUM_SCALE = 0x1p-13f, MV_SUM_UNSCALE = 0x1p13f;

// One 256-wide block of an activation row, by one warp (eight consecutive values per lane): digits, the block's scale, and
// the SUB-wide sums of the quantized values as f16 high and low parts.
struct MvX {
    float4 a, c;
    __device__ __forceinline__ void load(const float *__restrict__ src, bool want, int lane) { // a row not wanted counts as zero
        a = c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (want) {
            a = __ldg(reinterpret_cast<const float4 *>(src + lane * 8));
            c = __ldg(reinterpret_cast<const float4 *>(src + lane * 8) + 1);
        }
    }
};
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <int SUB>
__device__ __forceinline__ void mv_digits(const MvX &in, uint2 (&dig)[MV_NDIG], float &sx, __half &hi, __half &lo) {
    const float v[8] = {in.a.x, in.a.y, in.a.z, in.a.w, in.c.x, in.c.y, in.c.z, in.c.w};
    float amax = 0.f; // NaN if any value is: the block's scale, and with it the result, then is NaN too
#pragma unroll
    for (int j = 0; j < 8; j++) amax = max_nan(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float inv = amax > 0.f ? MV_QMAX / amax : 0.f;
    sx = amax * (1.0f / MV_QMAX);
    int sum = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t y[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int X = __float2int_rn(v[4 * h + j] * inv);
            sum += X;
            y[j] = (uint32_t)(X + 0x8080); // the two low digits become plain bytes plus 128
        }
        // byte d of the four values side by side; the 128 comes off again with the sign bit
        const uint32_t d2 = __byte_perm(__byte_perm(y[0], y[1], 0x40), __byte_perm(y[2], y[3], 0x40), 0x5410) ^ 0x80808080u;
        const uint32_t d1 = __byte_perm(__byte_perm(y[0], y[1], 0x51), __byte_perm(y[2], y[3], 0x51), 0x5410) ^ 0x80808080u;
        const uint32_t d0 = __byte_perm(__byte_perm(y[0], y[1], 0x62), __byte_perm(y[2], y[3], 0x62), 0x5410);
        if (h == 0) { dig[0].x = d0; dig[1].x = d1; dig[2].x = d2; }
        else { dig[0].y = d0; dig[1].y = d1; dig[2].y = d2; }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (SUB == 32) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const float sf = (float)sum * MV_SUM_SCALE;
    hi = __float2half_rn(sf);
    lo = __float2half_rn(sf - __half2float(hi));
}
// weight of digit d (most significant first)
__device__ __forceinline__ float mv_digit_weight(int d) { return d == 0 ? 65536.f : (d == 1 ? 256.f : 1.f); }

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
        mg = dg * (32.f * MV_SUM_UNSCALE);
        mG = dG * (32.f * MV_SUM_UNSCALE);
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

// ---- one pair -------------------------------------------------------------------------
// grid (ceil(n_out / 64), pairs), eight warps: row tile = warp % 4, K half = warp / 4.
// MMA columns 0-2: the digits; 3-7 repeat column 0 and are not read.
template <int DT>
__global__ void __launch_bounds__(MV_THREADS, 2)
mv_pair_kernel(const uint8_t *__restrict__ w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *__restrict__ x,
               int x_per_row, const uint32_t *__restrict__ ids, int top_k, float *__restrict__ out) {
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
    __half *sh = reinterpret_cast<__half *>(mv_smem + 3 * pitch);
    float *sxs = reinterpret_cast<float *>(mv_smem + 3 * pitch + 2 * bc * NS * 2);
    const int rt = warp & 3, ks = warp >> 2;
    const int rg = min(r_base + 16 * rt + g, n_out - 1), rG = min(r_base + 16 * rt + g + 8, n_out - 1);
    const uint8_t *wb = w + (size_t)e * expert_bytes;
    const uint8_t *pg = wb + (size_t)rg * row_bytes, *pG = wb + (size_t)rG * row_bytes;
    const float *xr = x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k;
    const int8_t *xcol = xc + (g < 3 ? g : 0) * pitch;
    const __half *scol = sh + (g == 1 ? bc * NS : 0); // column 0: high parts, column 1: low parts
    float yg = 0.f, yG = 0.f;
    for (int c0 = 0; c0 < nb; c0 += bc) {
        const int bn = min(bc, nb - c0);
        typename MvRaw<DT>::T raw;
        if (ks < bn) raw.load(pg + (size_t)(c0 + ks) * TS, pG + (size_t)(c0 + ks) * TS, t); // on its way while the activations are staged
        if (c0) __syncthreads(); // the previous digits have been read
        for (int b = warp; b < bn; b += MV_THREADS / 32) {
            uint2 dig[MV_NDIG];
            float sx;
            __half hi, lo;
            MvX in;
            in.load(xr + (size_t)(c0 + b) * QK_K, true, lane);
            mv_digits<SUB>(in, dig, sx, hi, lo);
#pragma unroll
            for (int d = 0; d < MV_NDIG; d++) *reinterpret_cast<uint2 *>(xc + d * pitch + b * QK_K + lane * 8) = dig[d];
            if ((lane & (SUB / 8 - 1)) == 0) {
                sh[b * NS + lane / (SUB / 8)] = hi;
                sh[bc * NS + b * NS + lane / (SUB / 8)] = lo;
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
            // lane t = 0 holds columns 0, 1 (and both halves of the sums), lane t = 1 column 2
            const float f0 = t == 0 ? 65536.f : (t == 1 ? 1.f : 0.f), f1 = t == 0 ? 256.f : 0.f, fm = t == 0 ? 1.f : 0.f, sx = sxs[b];
            yg += sx * (A.dg * (f0 * (float)al[0] + f1 * (float)al[1]) - A.mg * (fm * (cm[0] + cm[1])));
            yG += sx * (A.dG * (f0 * (float)al[2] + f1 * (float)al[3]) - A.mG * (fm * (cm[2] + cm[3])));
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
// grid (ceil(n_out / 64), ceil(pairs / 32)); the same warp layout.  The digits of 32 pairs are staged 1024 k at a time.
constexpr int MM_COLS = 32, MM_KC = 1024;
// bytes of a pair's digits: the columns of one load instruction (8 bytes a lane for Q4_K, 4 for Q6_K) cover distinct banks
template <int DT>
constexpr int MM_PITCH = MV_NDIG * MM_KC + (DT == LMOE_Q4_K ? 32 : 16);
template <int DT>
__global__ void __launch_bounds__(MV_THREADS, 2)
mv_multi_kernel(const uint8_t *__restrict__ w, int n_out, int k, const float *__restrict__ x, int x_per_row,
                const uint32_t *__restrict__ ids, int top_k, int pairs, float *__restrict__ out) {
    constexpr int SUB = DT == LMOE_Q4_K ? 32 : 16, NS = QK_K / SUB, BC = MM_KC / QK_K;
    constexpr int TS = DT == LMOE_Q4_K ? Q4K_BYTES : Q6K_BYTES;
    constexpr int SP = BC * NS + 8; // f16 sums of a pair and part, padded
    extern __shared__ __align__(16) uint8_t mv_smem[];
    int8_t *xc = reinterpret_cast<int8_t *>(mv_smem);                                                    // [pair][digit][k]
    __half *sh = reinterpret_cast<__half *>(mv_smem + MM_COLS * MM_PITCH<DT>);                           // [part][pair][SP]
    float *sxs = reinterpret_cast<float *>(mv_smem + MM_COLS * MM_PITCH<DT> + 2 * MM_COLS * SP * 2);     // [block][pair]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int p0 = blockIdx.y * MM_COLS, np = min(MM_COLS, pairs - p0), nb = k / QK_K;
    const int64_t row_bytes = (int64_t)nb * TS;
    const int r_base = blockIdx.x * MV_ROWS, rt = warp & 3, ks = warp >> 2;
    const int rg = min(r_base + 16 * rt + g, n_out - 1), rG = min(r_base + 16 * rt + g + 8, n_out - 1);
    const uint8_t *pg = w + (size_t)rg * row_bytes, *pG = w + (size_t)rG * row_bytes;
    float acc[MM_COLS / 8][4];
#pragma unroll
    for (int c = 0; c < MM_COLS / 8; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[c][i] = 0.f;
    for (int b0 = 0; b0 < nb; b0 += BC) {
        const int bn = min(BC, nb - b0);
        typename MvRaw<DT>::T raw;
        if (ks < bn) raw.load(pg + (size_t)(b0 + ks) * TS, pG + (size_t)(b0 + ks) * TS, t);
        __syncthreads(); // the previous chunk's digits have been read
        for (int i = warp; i < np * bn; i += MV_THREADS / 32) {
            const int p = i / bn, b = i - p * bn, pair = p0 + p;
            MvX in;
            in.load(x + ((size_t)(pair / top_k) * x_per_row + (x_per_row == 1 ? 0 : pair % top_k)) * k + (size_t)(b0 + b) * QK_K,
                    ids == nullptr || ids[pair] == 0u, lane);
            uint2 dig[MV_NDIG];
            float sx;
            __half hi, lo;
            mv_digits<SUB>(in, dig, sx, hi, lo);
#pragma unroll
            for (int d = 0; d < MV_NDIG; d++) *reinterpret_cast<uint2 *>(xc + p * MM_PITCH<DT> + d * MM_KC + b * QK_K + lane * 8) = dig[d];
            if ((lane & (SUB / 8 - 1)) == 0) {
                sh[p * SP + b * NS + lane / (SUB / 8)] = hi;
                sh[(MM_COLS + p) * SP + b * NS + lane / (SUB / 8)] = lo;
            }
            if (lane == 0) sxs[b * MM_COLS + p] = sx;
        }
        __syncthreads();
        for (int b = ks; b < bn; b += 2) {
            MvA<DT> A;
            A.unpack(raw, t);
            if (b + 2 < bn) raw.load(pg + (size_t)(b0 + b + 2) * TS, pG + (size_t)(b0 + b + 2) * TS, t);
#pragma unroll
            for (int c = 0; c < MM_COLS / 8; c++) {
                if (8 * c < np) { // columns past the last pair hold whatever was there: their results are not written
                    const int8_t *xp = xc + (8 * c + g) * MM_PITCH<DT> + b * QK_K;
                    float cm[4] = {0.f, 0.f, 0.f, 0.f}, tot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const __half *sp = sh + (h * MM_COLS + 8 * c + g) * SP + b * NS + 2 * t;
                        mma16816_acc(cm, A.f, *reinterpret_cast<const uint32_t *>(sp), NS == 16 ? *reinterpret_cast<const uint32_t *>(sp + 8) : 0u);
                    }
#pragma unroll
                    for (int d = 0; d < MV_NDIG; d++) {
                        int al[4] = {0, 0, 0, 0};
#pragma unroll
                        for (int i = 0; i < MvA<DT>::N; i++) {
                            int f[4];
                            A.mma(i, f, xp + d * MM_KC, t);
                            const int sg = A.sg(i), sG = A.sG(i);
                            al[0] += sg * f[0]; al[1] += sg * f[1]; al[2] += sG * f[2]; al[3] += sG * f[3];
                        }
#pragma unroll
                        for (int i = 0; i < 4; i++) tot[i] += mv_digit_weight(d) * (float)al[i];
                    }
                    const float2 sx = *reinterpret_cast<const float2 *>(sxs + b * MM_COLS + 8 * c + 2 * t);
                    acc[c][0] += sx.x * (A.dg * tot[0] - A.mg * cm[0]);
                    acc[c][1] += sx.y * (A.dg * tot[1] - A.mg * cm[1]);
                    acc[c][2] += sx.x * (A.dG * tot[2] - A.mG * cm[2]);
                    acc[c][3] += sx.y * (A.dG * tot[3] - A.mG * cm[3]);
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

template <int DT>
cudaError_t launch_mv(const uint8_t *w, int64_t expert_bytes, int n_expert, int n_out, int k, const float *x, int64_t pairs, int x_per_row,
                      const uint32_t *ids, int top_k, float *out, cudaStream_t s) {
    constexpr int NS = DT == LMOE_Q4_K ? 8 : 16;
    const unsigned gx = (unsigned)((n_out + MV_ROWS - 1) / MV_ROWS);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    // one matrix for all pairs: from four pairs on the columns of one unpacked super-block pay for the 32-pair staging
    if (n_expert == 1 && pairs >= 4) {
        constexpr int smem = MM_COLS * MM_PITCH<DT> + 2 * MM_COLS * (MM_KC / QK_K * NS + 8) * 2 + (MM_KC / QK_K) * MM_COLS * 4;
        static thread_local int c_dev = -1;
        if (dev != c_dev) {
            if ((e = cudaFuncSetAttribute(mv_multi_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
            c_dev = dev;
        }
        // grid.y is limited to 65535 groups
        const int64_t step = (int64_t)65535 * MM_COLS / top_k * top_k;
        for (int64_t p = 0; p < pairs; p += step) {
            const int64_t n = pairs - p < step ? pairs - p : step;
            mv_multi_kernel<DT><<<dim3(gx, (unsigned)((n + MM_COLS - 1) / MM_COLS)), MV_THREADS, smem, s>>>(
                w, n_out, k, x + (size_t)(p / top_k) * x_per_row * k, x_per_row, ids ? ids + p : nullptr, top_k, (int)n, out + (size_t)p * n_out);
        }
        return cudaGetLastError();
    }
    const int bc = k / QK_K < MV_PAIR_BLOCKS ? k / QK_K : MV_PAIR_BLOCKS;
    const int smem_pair = 3 * (bc * QK_K + 32) + 2 * bc * NS * 2 + bc * 4; // at most 27 KB
    // grid.y is limited to 65535: fold large pair counts over several launches
    const int64_t step = 65535 / top_k * top_k;
    for (int64_t p = 0; p < pairs; p += step) {
        const int64_t n = pairs - p < step ? pairs - p : step;
        mv_pair_kernel<DT><<<dim3(gx, (unsigned)n), MV_THREADS, smem_pair, s>>>(w, expert_bytes, n_expert, n_out, k,
                                                                                x + (size_t)(p / top_k) * x_per_row * k, x_per_row,
                                                                                ids ? ids + p : nullptr, top_k, out + (size_t)p * n_out);
    }
    return cudaGetLastError();
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
