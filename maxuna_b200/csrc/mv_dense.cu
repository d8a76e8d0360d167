// Many rows times ONE quantized matrix, as exact as the mat-vec kernels, on the 5th-generation tensor cores.
// Reference: the plain quantized product of `QMatMul`, src/ops/mv_id.rs:54-56, for a prompt chunk (the shared expert op by op).
//
// The operands are exact in f16, and so are the sums over a super-block in the f32 accumulators: integers of up to 2^24, whatever the values.  A Q4_K weight is its
// sub-block's integer scale times its integer, up to 63 x 15, and an activation five digits within +-64, in base 128, of a 30-bit integer (mv_digits.cuh):
// 256 x 945 x 64 = 0.92 x 2^24.  A Q6_K weight, up to 128 x 32, is in two parts with accumulators of their own, 8 x round(scale / 8) and the rest of the scale, up to 16 and 4 times 32, against
// four base-256 digits within +-128: 256 x 512 x 128 = 2^24.  (With both parts in one accumulator, in eighths, and four digits for Q4_K, operands of one sign lost up
// to five bits.)  The digits are columns of the B operand; the float factors, the weights of the digits and the Q4_K mins (a product of their own, against the sub-block sums in
// three exact parts) come in once a super-block, as in mv_multi_kernel, whose integer products need their scales after every 32 or 16 values.
// A super-block of 128 rows and 32 tokens takes 3.7 us (Q4_K; Q6_K 4.3 to 4.9), where its multiplies take 0.8 (1.2): the digits are made anew for every
// 128 rows, and with the storing of them and of the weights they fill the issue slots.  512 tokens [1024 x 3072] Q4_K 72 -> 49 us,
// [3072 x 1024] Q6_K 115 -> 66, with the same error against 64 bits.
#include "common.cuh"
#include "kquant.cuh"
#include "mv_digits.cuh"
#include "tc.cuh"

namespace {

constexpr int MD_ROWS = 128, MD_TOK = 32; // a block's weight rows and tokens
constexpr int MD_WORK = 512, MD_THREADS = MD_WORK + 32; // sixteen warps make operands and take results, one issues
constexpr int MD_Q6_WORDS = 53, MD_Q6_PITCH = 55;       // words that hold a 210-byte block at an even address; of a row of the staged blocks
constexpr int MD_TILE = 128 * 128; // an operand tile of 128 rows x 64 values
constexpr int MD_SUMS = 3 * MD_TOK * 128;

template <int DT>
struct MdCfg {
    static constexpr bool Q4 = DT == LMOE_Q4_K;
    static constexpr int NDIG = Q4 ? 5 : MV_NDIG, COLS = NDIG * MD_TOK; // digits of an activation; column 32 d + i: digit d of token i
    static constexpr int B_TILE = COLS * 128;
    static constexpr int O_LOW = 4 * MD_TILE, O_B = (Q4 ? 4 : 8) * MD_TILE, O_MINS = O_B + 4 * B_TILE, O_SUMS = O_MINS + MD_TILE;
    static constexpr int O_RAW = O_MINS; // Q6_K: the super-block's bytes of all rows
    static constexpr int SMEM = (Q4 ? O_SUMS + MD_SUMS : O_RAW + MD_ROWS * MD_Q6_PITCH * 4) + 1024;
};

__device__ __forceinline__ uint32_t md_sub(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t md_twice(float v) { // f16 pair (v, v)
    const uint32_t h = __half_as_ushort(__float2half_rn(v));
    return h | h << 16;
}
__device__ __forceinline__ void md_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a),
                 "l"(b), "r"(idesc), "r"(accum) : "memory");
}
// A Q4_K activation as fields of 7, 7, 7, 7 and 4 bits from the lowest on, made positive by 64 and 8: f[p] holds, for the two values of pair p, fields 0 and 1 and the upper
// two bits of the last one, f[4 + p] fields 2 and 3 and its lower two.
__device__ __forceinline__ void md_fields(const int (&X)[8], uint32_t (&f)[8]) {
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const int i = (p & 1) + 4 * (p >> 1);
        const uint32_t a = (uint32_t)X[i] + 0x88102040u, c = (uint32_t)X[i + 2] + 0x88102040u, ah = a >> 14, ch = c >> 14;
        f[p] = __byte_perm((a & 0x3FFFu) | (ah >> 2 & 0xC000u), (c & 0x3FFFu) | (ch >> 2 & 0xC000u), 0x5410);
        f[4 + p] = __byte_perm(ah, ch, 0x5410);
    }
}
// place of 16-byte chunk c of row r of an operand tile
__device__ __forceinline__ int md_at(int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); }

// Sixteen warps make the operands of a super-block, another one issues its multiplies, and while these run the sixteen take the super-block before out of tensor
// memory and turn the next one's activations into digits (registers).  (With the roles given to different warps each of them waits for its
// instructions: 512 tokens [1024 x 3072] Q4_K 59 us.)
template <int DT>
__global__ void __launch_bounds__(MD_THREADS, 1)
mv_dense_kernel(const uint8_t *__restrict__ w, int n_out, int k, const float *__restrict__ x, int x_per_row, const uint32_t *__restrict__ ids, int top_k,
                int pairs, float *__restrict__ out) {
    using C = MdCfg<DT>;
    constexpr int TS = C::Q4 ? Q4K_BYTES : Q6K_BYTES, SUB = C::Q4 ? 32 : 16;
    extern __shared__ uint8_t md_raw[];
    uint8_t *smem = md_raw + (0u - s32(md_raw) & 1023u); // (an offset: the compiler goes on knowing it as shared memory)
    uint8_t *a_st = smem, *b_st = smem + C::O_B, *mins = smem + C::O_MINS, *sums = smem + C::O_SUMS;
    __shared__ uint64_t done;
    __shared__ float sxs[4][MD_TOK];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = k / QK_K;
    const int r0 = blockIdx.x * MD_ROWS, p0 = blockIdx.y * MD_TOK;
    const int64_t row_bytes = (int64_t)nb * TS;
    if (tid == 0) {
        mb_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MD_WORK / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (C::Q4) { // the second half of the mins' 16 k is zero
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        if (tid < MD_ROWS) *reinterpret_cast<uint4 *>(mins + md_at(tid, 1)) = zero;
        else if (tid < MD_ROWS + 3 * MD_TOK) *reinterpret_cast<uint4 *>(sums + md_at(tid - MD_ROWS, 1)) = zero;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_begin();
    // weights: thread = (row, 64-k tile); activations: a warp has tokens warp and warp + 16; results: the same row, eight tokens
    const int r = tid & (MD_ROWS - 1), j = (tid >> 7) & 3, q = warp & 3, part8 = (warp >> 2) & 3;
    const int row = min(r0 + r, n_out - 1);
    int src[2]; // rows of x, or -1
#pragma unroll
    for (int v = 0; v < 2; v++) {
        const int p = p0 + (warp & 15) + 16 * v;
        const bool want = p < pairs && (ids == nullptr || ids[p] == 0u); // another id names no matrix of this stack: a zero row
        src[v] = want ? (x_per_row == 1 ? p / top_k : p) : -1;           // (x_per_row is 1 or top_k)
    }
    MvX in[2];
    uint4 hdr, qa, qb;          // Q4_K: this tile's words
    auto load_x = [&](int b) {
#pragma unroll
        for (int v = 0; v < 2; v++) in[v].load(x + (size_t)max(src[v], 0) * k + b * QK_K, src[v] >= 0, lane);
    };
    auto load_w = [&](int b) {
        const uint8_t *blk = w + (row * row_bytes + (int64_t)b * TS);
        if (C::Q4) {
            hdr = __ldg(reinterpret_cast<const uint4 *>(blk));
            qa = __ldg(reinterpret_cast<const uint4 *>(blk) + 1 + 2 * j);
            qb = __ldg(reinterpret_cast<const uint4 *>(blk) + 2 + 2 * j);
        } else { // whole rows, a word a lane (word by word of its own row a thread took 14 thousand cycles a super-block)
            for (int i = 0; i < MD_ROWS / 16; i++) {
                const int rr = warp * (MD_ROWS / 16) + i;
                const uint8_t *g = w + (size_t)min(r0 + rr, n_out - 1) * row_bytes + (size_t)b * TS;
                const uint32_t *g4 = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(g) & ~(uintptr_t)3);
                uint32_t *to = reinterpret_cast<uint32_t *>(smem + C::O_RAW) + rr * MD_Q6_PITCH;
#pragma unroll
                for (int o = 0; o < 64; o += 32)
                    if (lane + o < MD_Q6_WORDS) { // (of the last word of a block at a word's start only two bytes are the block's, and may be the matrix's last)
                        const uint32_t n = lane + o == MD_Q6_WORDS - 1 && !(reinterpret_cast<uintptr_t>(g) & 2) ? 2u : 4u;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s32(to + lane + o)), "l"(g4 + lane + o), "r"(n) : "memory");
                    }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    float acc[8], odd[8];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = odd[i] = 0.f;
    auto take = [&](int b, float d, float m) { // of super-block b: d, dmin of the row
        const uint32_t t0 = tmem + 256u * (b & 1) + ((uint32_t)(32 * q) << 16) + 8u * part8;
        constexpr int MORE = C::Q4 ? MV_PARTS : C::NDIG; // parts of the mins' sums, or the low parts of the weights
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            float tot[4], off[4];
            { // digits from the least significant on, so that only the last addition rounds at the size of the sum
                uint32_t v[C::NDIG][4];
#pragma unroll
                for (int e = 0; e < C::NDIG; e++) tc_ld4(t0 + MD_TOK * e + h, v[e]);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    tot[i] = __uint_as_float(v[C::NDIG - 1][i]);
#pragma unroll
                    for (int e = C::NDIG - 2; e >= 0; e--)
                        tot[i] = __fmaf_rn(C::Q4 ? (float)(1 << 7 * (C::NDIG - 1 - e)) : mv_digit_weight(e), __uint_as_float(v[e][i]), tot[i]);
                }
            }
            {
                uint32_t v[MORE][4];
#pragma unroll
                for (int e = 0; e < MORE; e++) tc_ld4(t0 + C::COLS + MD_TOK * e + h, v[e]);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    off[i] = __uint_as_float(v[MORE - 1][i]);
#pragma unroll
                    for (int e = MORE - 2; e >= 0; e--)
                        off[i] = C::Q4 ? __uint_as_float(v[e][i]) + off[i] : __fmaf_rn(mv_digit_weight(e), __uint_as_float(v[e][i]), off[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                // (two sums of half of the super-blocks, in turn, round less than one of all)
                const float o = acc[h + i] + sxs[b & 3][8 * part8 + h + i] * (C::Q4 ? d * tot[i] - m * off[i] : d * __fmaf_rn(8.f, tot[i], off[i]));
                acc[h + i] = odd[h + i];
                odd[h + i] = o;
            }
        }
        tc_fence_before();
    };
    bool ok = true;
    if (warp == MD_WORK / 32) {
        const bool el = elect_one();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(C::COLS >> 3) << 17) | ((uint32_t)(MD_ROWS >> 4) << 24);
        const uint32_t idesc_m = (1u << 4) | ((uint32_t)(3 * MD_TOK >> 3) << 17) | ((uint32_t)(MD_ROWS >> 4) << 24);
        const uint64_t ad = umma_desc(s32(a_st)), bd = umma_desc(s32(b_st)), md = umma_desc(s32(mins)), sd = umma_desc(s32(sums));
        for (int b = 0; b < nb; b++) {
            __syncthreads(); // the operands are there
            tc_fence_after();
            const uint32_t d = tmem + 256u * (b & 1);
            if (el) {
                if (C::Q4) md_mma(d + C::COLS, md, sd, idesc_m, 0u);
#pragma unroll
                for (uint32_t t = 0; t < 4; t++) {
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) {
                        const uint64_t bt = bd + t * (C::B_TILE >> 4) + 2 * kk;
                        md_mma(d, ad + t * (MD_TILE >> 4) + 2 * kk, bt, idesc, t | kk);
                        if (!C::Q4) md_mma(d + C::COLS, ad + ((C::O_LOW + t * MD_TILE) >> 4) + 2 * kk, bt, idesc, t | kk);
                    }
                }
                tc_commit<1>(&done);
            }
            __syncwarp();
        }
        ok = mb_wait(&done, (uint32_t)(nb - 1) & 1u); // none is in flight when the tensor memory is given back
    }
    float d = 0.f, m = 0.f;
    if (warp < MD_WORK / 32) {
        load_x(0);
        load_w(0);
    }
    for (int b = 0; b < nb && warp < MD_WORK / 32; b++) {
        uint32_t dig[2][8]; // Q4_K: words (0 2), (1 3), (4 6), (5 7) of the lower 14 bits and of the others, see md_fields; Q6_K: two words a digit
        float sx[2];
        __half sub[2][MV_PARTS];
#pragma unroll
        for (int v = 0; v < 2; v++) {
            int X[8];
            mv_integers<SUB>(in[v], X, sx[v], sub[v]);
            if constexpr (C::Q4) {
                md_fields(X, dig[v]);
            } else {
                uint2 d[MV_NDIG];
                mv_bytes(X, d);
#pragma unroll
                for (int e = 0; e < MV_NDIG; e++) dig[v][2 * e] = d[e].x, dig[v][2 * e + 1] = d[e].y;
            }
        }
        if (b + 1 < nb) load_x(b + 1);
        if (!C::Q4) asm volatile("cp.async.wait_group 0;\n\tbar.sync 1, 512;" ::: "memory"); // all rows' bytes are there
        if (b && ok) ok = mb_wait(&done, (uint32_t)(b - 1) & 1u); // the operands of the super-block before have been multiplied
        tc_fence_after();
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int i = warp + 16 * v;
            uint8_t *to = b_st + (lane >> 3) * C::B_TILE;
            auto put = [&](int d, const uint32_t (&h)[4]) { *reinterpret_cast<uint4 *>(to + md_at(MD_TOK * d + i, lane & 7)) = make_uint4(h[0], h[1], h[2], h[3]); };
            // f16 pairs in the order of the weights' chunks: 0 2 1 3 4 6 5 7
            uint32_t h[4];
            if constexpr (C::Q4) {
                const uint32_t seven = 0x007F007Fu, off = 0x64406440u;
#pragma unroll
                for (int d = 1; d < 5; d++) {
#pragma unroll
                    for (int p = 0; p < 4; p++) h[p] = md_sub(and_or((d < 3 ? dig[v][4 + p] : dig[v][p]) >> ((d & 1) ? 7 : 0), seven, 0x64006400u), off);
                    put(d, h);
                }
#pragma unroll
                for (int p = 0; p < 4; p++)
                    h[p] = md_sub(and_or(dig[v][p] >> 12, 0x000C000Cu, and_or(dig[v][4 + p] >> 14, 0x00030003u, 0x64006400u)), 0x64086408u);
                put(0, h);
            } else {
#pragma unroll
                for (int d = 0; d < MV_NDIG; d++) {
                    const uint32_t lo = dig[v][2 * d] ^ 0x80808080u, hi = dig[v][2 * d + 1] ^ 0x80808080u, one = 0x64646464u, off = 0x64806480u;
                    h[0] = md_sub(__byte_perm(lo, one, 0x4240), off), h[1] = md_sub(__byte_perm(lo, one, 0x4341), off);
                    h[2] = md_sub(__byte_perm(hi, one, 0x4240), off), h[3] = md_sub(__byte_perm(hi, one, 0x4341), off);
                    put(d, h);
                }
            }
            if (C::Q4 && (lane & 3) == 0) {
#pragma unroll
                for (int h = 0; h < MV_PARTS; h++)
                    *reinterpret_cast<__half *>(sums + md_at(MD_TOK * h + i, 0) + 2 * (lane >> 2)) = sub[v][h];
            }
            if (lane == 0) sxs[b & 3][i] = sx[v];
        }
        uint8_t *a = a_st + j * MD_TILE;
        int rr = r;
        asm volatile("" : "+r"(rr)); // the places of the eight stores are worked out here and not kept in registers
        uint16_t d6 = 0;
        if constexpr (C::Q4) {
            uint32_t scs[2], mn[2];
            q4k_unpack_scales(hdr.y, hdr.z, hdr.w, scs[0], scs[1], mn[0], mn[1]);
            if (j == 0) {
                const uint32_t one = 0x64646464u, off = 0x64006400u;
                *reinterpret_cast<uint4 *>(mins + md_at(r, 0)) =
                    make_uint4(md_sub(__byte_perm(mn[0], one, 0x4140), off), md_sub(__byte_perm(mn[0], one, 0x4342), off),
                               md_sub(__byte_perm(mn[1], one, 0x4140), off), md_sub(__byte_perm(mn[1], one, 0x4342), off));
            }
            const uint32_t pair = md_sub(__byte_perm((j & 2) ? scs[1] : scs[0], 0x64646464u, (j & 1) ? 0x4342u : 0x4140u), 0x64006400u);
            const uint32_t v[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t s = __byte_perm(pair, 0u, h ? 0x3232u : 0x1010u), c0 = h2_mul(s, 0xE400E400u); // - 1024 scales
#pragma unroll
                for (int c = 0; c < 4; c++) { // (1024 + q) scale - 1024 scale: exact
                    const uint32_t u0 = v[2 * c] >> (4 * h), u1 = v[2 * c + 1] >> (4 * h);
                    *reinterpret_cast<uint4 *>(a + md_at(rr, 4 * h + c)) =
                        make_uint4(h2_fma(and_or(u0, 0x000F000Fu, 0x64006400u), s, c0), h2_fma(and_or(u0 >> 8, 0x000F000Fu, 0x64006400u), s, c0),
                                   h2_fma(and_or(u1, 0x000F000Fu, 0x64006400u), s, c0), h2_fma(and_or(u1 >> 8, 0x000F000Fu, 0x64006400u), s, c0));
                }
            }
        } else {
            // half j / 2, groups 2 (j % 2) + h
            const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(w + (row * row_bytes + (int64_t)b * TS)) & 2) * 8u;
            const uint32_t *st = reinterpret_cast<const uint32_t *>(smem + C::O_RAW) + r * MD_Q6_PITCH;
            auto word = [&](int i) { return __funnelshift_r(st[i], st[i + 1], off); }; // bytes 4 i .. 4 i + 3 of the block
            const uint32_t scs = word(48 + 2 * (j >> 1) + (j & 1));
            d6 = (uint16_t)(off ? st[52] >> 16 : st[52]);
#pragma unroll
            for (int h = 0; h < 2; h++) { // group 2 (j % 2) + h: its two scales are side by side
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int s = (int8_t)(scs >> (16 * h + (c < 2 ? 0 : 8)));
                    const uint32_t hi = md_twice((float)((s + 4) >> 3)), lo = md_twice((float)(s - ((s + 4) & ~7)));
                    uint32_t e[4];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const uint32_t ql = word(16 * (j >> 1) + 8 * h + 2 * c + i) >> (4 * (j & 1));
                        const uint32_t t = (word(32 + 8 * (j >> 1) + 2 * c + i) >> (4 * (j & 1) + 2 * h) & 0x03030303u) << 4;
                        const uint32_t q6 = and_or(ql, 0x0F0F0F0Fu, t);
                        e[2 * i] = md_sub(__byte_perm(q6, 0x64646464u, 0x4240), 0x64206420u);
                        e[2 * i + 1] = md_sub(__byte_perm(q6, 0x64646464u, 0x4341), 0x64206420u);
                    }
                    *reinterpret_cast<uint4 *>(a + md_at(rr, 4 * h + c)) = make_uint4(h2_mul(e[0], hi), h2_mul(e[1], hi), h2_mul(e[2], hi), h2_mul(e[3], hi));
                    *reinterpret_cast<uint4 *>(a + C::O_LOW + md_at(rr, 4 * h + c)) = make_uint4(h2_mul(e[0], lo), h2_mul(e[1], lo), h2_mul(e[2], lo), h2_mul(e[3], lo));
                }
            }
        }
        const float d_now = C::Q4 ? lmoe_h2f((uint16_t)(hdr.x & 0xffff)) : lmoe_h2f(d6);
        const float m_now = C::Q4 ? lmoe_h2f((uint16_t)(hdr.x >> 16)) * MV_SUM_UNSCALE : 0.f;
        if (C::Q4 && b + 1 < nb) load_w(b + 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (!C::Q4 && b + 1 < nb) load_w(b + 1); // (all have read this one's bytes)
        if (b) take(b - 1, d, m);
        d = d_now;
        m = m_now;
    }
    if (warp < MD_WORK / 32) {
        if (ok) ok = mb_wait(&done, (uint32_t)(nb - 1) & 1u);
        tc_fence_after();
        take(nb - 1, d, m);
    }
    const int bad = __syncthreads_or(!ok);
    const int ro = r0 + 32 * q + lane;
    if (ro < n_out && warp < MD_WORK / 32) {
#pragma unroll
        for (int i = 0; i < 8; i++) { // (a wait that ran out leaves NaN, not a wrong number)
            const int p = p0 + 8 * part8 + i;
            if (p < pairs) out[(size_t)p * n_out + ro] = bad ? __int_as_float(0x7fffffff) : acc[i] + odd[i];
        }
    }
    if (warp == MD_WORK / 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

template <int DT>
cudaError_t launch_dense(const uint8_t *w, int n_out, int k, const float *x, int64_t pairs, int x_per_row, const uint32_t *ids, int top_k, float *out,
                         cudaStream_t s) {
    static thread_local int c_dev = -1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev != c_dev) {
        if ((e = cudaFuncSetAttribute(mv_dense_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, MdCfg<DT>::SMEM)) != cudaSuccess) return e;
        c_dev = dev;
    }
    // grid.y is limited to 65535 groups
    const int64_t step = (int64_t)65535 * MD_TOK / top_k * top_k;
    for (int64_t p = 0; p < pairs; p += step) {
        const int64_t n = pairs - p < step ? pairs - p : step;
        launch_pdl(mv_dense_kernel<DT>, dim3((unsigned)((n_out + MD_ROWS - 1) / MD_ROWS), (unsigned)((n + MD_TOK - 1) / MD_TOK)), MD_THREADS, MdCfg<DT>::SMEM, s,
                   w, n_out, k, x + (size_t)(p / top_k) * x_per_row * k, x_per_row, ids ? ids + p : nullptr, top_k, (int)n, out + (size_t)p * n_out);
    }
    return cudaGetLastError();
}

} // namespace

// out[pair][n_out] = the matrix times the pair's row of x; ids as in launch_mul_mv_id for a stack of one.
cudaError_t launch_mv_dense(int dtype, const uint8_t *w, int n_out, int k, const float *x, int64_t pairs, int x_per_row, const uint32_t *ids, int top_k,
                            float *out, cudaStream_t s) {
    return dtype == LMOE_Q4_K ? launch_dense<LMOE_Q4_K>(w, n_out, k, x, pairs, x_per_row, ids, top_k, out, s)
                              : launch_dense<LMOE_Q6_K>(w, n_out, k, x, pairs, x_per_row, ids, top_k, out, s);
}
