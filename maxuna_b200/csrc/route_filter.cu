// Routing of long prompts: the tensor core says which experts can be among a token's top_k, and only those get the specified
// f32 logit.  Ids and weights are those of route.cu to the bit.
// Reference: `route_logits` and `route_from_logits`, src/moe.rs:84-119.
//
// The specified logits (route_math.cuh) are f32 products in a fixed order: for 16384 tokens, 256 experts and hidden 3072 they and the selection
// take 730 us at half of the f32 rate, for 2048 tokens 115.  This takes 290 and 60: 5 for the router's f16 image, 42 / 13 for the approximate product
// (16384 tokens: the tokens from memory at 4.8 TB/s), 240 / 38 for the rest (the router rows from the L2 cache).  A product of the operands rounded to f16 differs from it by at most
//   |x| |w| (2^-10 + 2^-22 + 17/16 hidden 2^-23 + 2^-18) + 2^-25 sqrt(hidden) (|x| + |w|)
// (2^-11 for the rounding of either operand by Cauchy's inequality; the tensor core adds sixteen products to a sum at a time, each of the seventeen
// cut, at worst, at the last of 24 bits of the largest of them; 2^-18 for the sum of the parts and for the specified sum, each a chain of at most 39 roundings; the last
// term for values below the f16 range), so it bounds every score, and an expert whose
// upper bound is below the top_k-th largest lower bound is out.  13 of 256 experts are left for a token of random normal values and weights, 12 with
// weights ten times as large, 39 where eight of the 3072 channels are a hundred times the others and their weights a hundredth.  A token with a bound that is not
// finite (an operand beyond the f16 range, an infinity, NaN) keeps all its experts, as do scores that all tie, but for a row of zeros, whose logits are known.
// How many are left hangs on the data, so it is counted: up to a quarter of the experts on the average of a block's tokens, and one token that keeps all, the block
// computes their logits itself; beyond, the router rows that it reads for every four tokens take longer than the tiled f32 product does, and the tokens that keep
// too many go to a kernel of that product.
// A block's forward, hidden 3072, 256 experts of 256, 2048 tokens (3072 tokens), f32 routing alone 409 us (534): 345 (468) at 13 left, 364 (499) at 24, 384 (535) at 39,
// 466 (635) at 97, 447 (606) at 165 and 426 (591) at all 256; with all computed in the blocks 20 to 35 % more than the f32 routing from 97 left on.
#include <math.h>
#include <type_traits>

#include "fused.cuh"
#include "route_math.cuh"
#include "route_tile.cuh"
#include "tc.cuh"

namespace {

constexpr int RF_A_BYTES = 128 * 128; // 128 tokens x 64 values as f16
constexpr int RF_STAGES = 4;
constexpr int RF_SPLITS = 4; // most parts that hidden is cut into
constexpr int RF_AHEAD = 3; // stages whose words a producing thread has in flight

// The router as f16 in the order of the B operand's stages (64 values of all experts: a 128-byte-swizzled tile), and its rows' norms.
// A block per expert.  clear: the call's control words; done: route_dense_kernel's counts.
__global__ void __launch_bounds__(128) route_prep_kernel(const float *__restrict__ router, int hidden, int n_expert, uint8_t *__restrict__ img,
                                                         float *__restrict__ wnorm, uint32_t *__restrict__ clear, uint32_t *__restrict__ done, int tiles) {
    pdl_begin();
    const int e = blockIdx.x;
    if (e == 0 && threadIdx.x < LMOE_CONTROL_WORDS) clear[threadIdx.x] = 0u;
    for (int i = e * 128 + threadIdx.x; i < tiles; i += n_expert * 128) done[i] = 0u;
    const float4 *w = reinterpret_cast<const float4 *>(router + (size_t)e * hidden);
    float ss = 0.f;
    for (int ci = threadIdx.x; ci < hidden / 8; ci += 128) {
        const float4 a = __ldg(w + 2 * ci), b = __ldg(w + 2 * ci + 1);
        ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
        __align__(16) __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w), __floats2half2_rn(b.x, b.y),
                                      __floats2half2_rn(b.z, b.w)};
        *reinterpret_cast<uint4 *>(img + ((size_t)(ci >> 3) * n_expert + e) * 128 + (((ci & 7) ^ (e & 7)) << 4)) = *reinterpret_cast<const uint4 *>(h);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    __shared__ float part[4];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) wnorm[e] = sqrtf(part[0] + part[1] + part[2] + part[3]);
}

// Approximate logits of TM tokens (the M of the multiplies is 128; rows past the last token are whatever lies there, and nothing reads
// their results) and all experts, over part blockIdx.y of hidden (the parts' results follow one another, t x n_expert each): eight warps round the tokens to f16 and put them into the A stages, warp 8
// issues the multiplies, warp 9 copies the B stages, warps 0-3 take the results out of tensor memory.  xss: the tokens' squared norms, by part.
// What a block reads bounds it, some 60 bytes a cycle and SM from the L2 cache: for few tokens the parts of hidden cut that, where parts of the experts would
// read the tokens again (2048 tokens: 64 blocks of half of the experts 21 us, 128 of a quarter of hidden 13).
template <int TM>
__global__ void __launch_bounds__(320, 1) route_approx_kernel(const float *__restrict__ x, const uint8_t *__restrict__ img, int t, int hidden, int n_expert,
                                                              float *__restrict__ logits, float *__restrict__ xss, uint32_t *__restrict__ flag) {
    constexpr int GROUPS = TM == 64 ? 2 : 1; // groups of producing warps, which take the stages in turn
    extern __shared__ uint8_t rf_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(rf_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t a_full[RF_STAGES], b_full[RF_STAGES], empty[RF_STAGES], done;
    __shared__ uint32_t tmem_slot;
    __shared__ float sums[TM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, steps = hidden / 64 / (int)gridDim.y, s00 = (int)blockIdx.y * steps;
    const int t0 = blockIdx.x * TM, nt = min(TM, t - t0);
    const uint32_t b_bytes = (uint32_t)n_expert * 128u;
    uint8_t *a_st = smem, *b_st = smem + RF_STAGES * RF_A_BYTES;
    if (tid == 0) {
        for (int s = 0; s < RF_STAGES; s++) {
            mb_init(&a_full[s], 8 / GROUPS);
            mb_init(&b_full[s], 1);
            mb_init(&empty[s], 1);
        }
        mb_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&tmem_slot)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_begin();
    bool ok = true;
    if (warp < 8) {
        constexpr int THREADS = 256 / GROUPS, RS = THREADS / 8, NC = TM / RS; // 8-value chunks of a thread and stage: one of rows r0, r0 + RS, ...
        const int grp = tid / THREADS, ch = tid & 7, r0 = tid % THREADS >> 3;
        const float4 *src[NC];
        uint8_t *dst[NC];
        float ss[NC];
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int r = r0 + RS * i;
            src[i] = reinterpret_cast<const float4 *>(x + (size_t)(t0 + min(r, nt - 1)) * hidden) + 16 * s00 + 2 * ch;
            dst[i] = a_st + r * 128 + ((ch ^ (r & 7)) << 4);
            ss[i] = 0.f;
        }
        float4 v[RF_AHEAD][NC][2];
        auto load = [&](int u, int s) {
#pragma unroll
            for (int i = 0; i < NC; i++)
#pragma unroll
                for (int h = 0; h < 2; h++) v[u][i][h] = s < steps ? __ldg(src[i] + 16 * s + h) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
#pragma unroll
        for (int u = 0; u < RF_AHEAD; u++) load(u, grp + GROUPS * u);
        uint32_t st = grp, ph = 0;
        for (int s0 = grp; s0 < steps && ok; s0 += GROUPS * RF_AHEAD) {
#pragma unroll
            for (int u = 0; u < RF_AHEAD; u++) {
                if (s0 + GROUPS * u >= steps) break;
                ok &= mb_wait(&empty[st], ph ^ 1);
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    const float4 a = v[u][i][0], b = v[u][i][1];
                    ss[i] += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
                    __align__(16) __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w), __floats2half2_rn(b.x, b.y),
                                                  __floats2half2_rn(b.z, b.w)};
                    *reinterpret_cast<uint4 *>(dst[i] + st * RF_A_BYTES) = *reinterpret_cast<const uint4 *>(h);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mb_arrive(&a_full[st]);
                if ((st += GROUPS) >= RF_STAGES) { st -= RF_STAGES; ph ^= 1; }
                load(u, s0 + GROUPS * (u + RF_AHEAD));
            }
        }
        { // (the groups' shares meet in shared memory)
#pragma unroll
            for (int i = 0; i < NC; i++) {
#pragma unroll
                for (int o = 4; o; o >>= 1) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
                if (GROUPS == 2 && grp == 1 && ch == 0) sums[r0 + RS * i] = ss[i];
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int r = r0 + RS * i;
                if (grp == 0 && ch == 0 && r < nt) xss[(size_t)blockIdx.y * t + t0 + r] = GROUPS == 2 ? ss[i] + sums[r] : ss[i];
            }
        }
        if (warp < 4) { // a lane is a token
            ok &= mb_wait(&done, 0);
            tc_fence_after();
            const int r = 32 * warp + lane;
            float *dstl = logits + ((size_t)blockIdx.y * t + t0 + r) * n_expert;
            if (32 * warp < nt)
                for (int c = 0; c < n_expert; c += 16) {
                    uint32_t o[16];
                    tc_ld16(tmem + ((uint32_t)(32 * warp) << 16) + c, o);
                    tc_wait_ld();
                    if (r < nt) {
#pragma unroll
                        for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(dstl + c + 4 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                    }
                }
            tc_fence_before();
        }
    } else if (warp == 8) {
        const bool el = elect_one();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n_expert >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        uint32_t st = 0, ph = 0;
        for (int s = 0; s < steps && ok; s++) {
            ok &= mb_wait(&b_full[st], ph);
            ok &= mb_wait(&a_full[st], ph);
            tc_fence_after();
            if (el) {
                const uint64_t ad = umma_desc(s32(a_st + st * RF_A_BYTES)), bd = umma_desc(s32(b_st + st * b_bytes));
#pragma unroll
                for (int kk = 0; kk < 4; kk++)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem), "l"(ad + 2 * kk), "l"(bd + 2 * kk), "r"(idesc),
                                 "r"((uint32_t)(s | kk)) : "memory");
                tc_commit<1>(&empty[st]);
            }
            __syncwarp();
            if (++st == RF_STAGES) { st = 0; ph ^= 1; }
        }
        if (el) tc_commit<1>(&done);
        __syncwarp();
        ok &= mb_wait(&done, 0); // none is in flight when the tensor memory is given back
    } else if (warp == 9) {
        const bool el = elect_one();
        uint32_t st = 0, ph = 0;
        for (int s = 0; s < steps && ok; s++) {
            ok &= mb_wait(&empty[st], ph ^ 1);
            if (el) {
                mb_expect_tx(&b_full[st], b_bytes);
                bulk_g2s(b_st + st * b_bytes, img + (size_t)(s00 + s) * n_expert * 128, b_bytes, &b_full[st]);
            }
            __syncwarp();
            if (++st == RF_STAGES) { st = 0; ph ^= 1; }
        }
        // the copies have landed: slots below st in the present turn of the ring, the others in the turn before
        for (uint32_t i = 0; i < RF_STAGES; i++) {
            const bool here = mb_wait(&b_full[i], i < st ? ph : ph ^ 1);
            ok &= here;
            if (!here) break;
        }
    }
    if (!ok && lane == 0 && atomicCAS(flag, 0u, (uint32_t)LMOE_FLAG_WAIT_TIMEOUT) == 0u) {
        flag[1] = 0x2000u + warp;
        flag[2] = blockIdx.x;
    }
    if (__syncthreads_or(!ok)) // a wait ran out: no bound is known, and the tokens keep all their experts
        for (int i = tid; i < nt * n_expert; i += 320) logits[((size_t)blockIdx.y * t + t0) * n_expert + i] = __int_as_float(0x7fffffff);
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

// The specified logits of the experts that the approximate ones leave, then the selection: a block of TB tokens, whose rows lie in
// shared memory.  The experts left for any of them are taken in turn by sixteen warps, each router row once for up to
// four tokens: some 150 rows for some 210 logits of sixteen tokens.  The rows from the L2 cache are what bounds it (16384 tokens: 1.8 GB; with each piece
// of a row waited for before the next is asked for 424 us; with sixteen exact sigmoids a lane for the bounds and selection by rounds 297; so 240).
constexpr int RV_WARPS = 16, RV_TOKENS = 4, RV_PIECE = 8;
constexpr uint32_t RV_OUT = 0xffa5a5a5u; // in place of the logit of an expert that is out: a NaN that no operation results in

// A bound below (side = -1) or above (1) of the specified sigmoid (route_math.cuh) of v, from the hardware's exponential and reciprocal.  These are
// off by 2 + 1.2 |v| units in the last place (2^-23) of the exponential, which count (1 - sigmoid) times, and by three of the quotient; the specified one, which stops at
// |v| = 87, by less.  The last term is for values below the normal range and for quotients that the hardware's division gives as 0.
__device__ __forceinline__ float route_bound(float v, float side) {
    const float a = fminf(fmaxf(-v, -88.f), 88.f), p = __fdividef(1.f, 1.f + __expf(a));
    return p + side * (p * (8e-7f + (1e-6f + 2e-7f * fabsf(a)) * (1.f - p)) + 1e-37f);
}

// As in route_select_kernel, from a token's logits in shared memory; the experts that are out do not exist.
template <int PER>
__device__ __forceinline__ void route_select_token(float *probs, const float *__restrict__ bias, int n_expert, int top_k, float scale, int norm, uint32_t *ids_row,
                                                   float *w_row, int lane) {
    uint32_t key[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int e = lane + 32 * j;
        key[j] = 0u;
        if (e < n_expert) {
            const float v = probs[e];
            if (__float_as_uint(v) != RV_OUT) {
                const float p = lmoe_sigmoid_fixed(v);
                probs[e] = p;
                key[j] = lmoe_score_key(bias ? __fadd_rn(p, __ldg(bias + e)) : p);
            }
        }
    }
    __syncwarp();
    lmoe_warp_select_keys<PER>(key, probs, top_k, scale, norm, ids_row, w_row, lane);
}

template <int TB, int PER>
__global__ void __launch_bounds__(RV_WARPS * 32, 1)
route_verify_kernel(const float *__restrict__ router, const float *__restrict__ x, const float *__restrict__ bias, const float *__restrict__ approx,
                    const float *__restrict__ xss, int splits, const float *__restrict__ wnorm, int t, int hidden, int n_expert, int top_k, float scale, int norm,
                    uint32_t *__restrict__ ids, float *__restrict__ weights, int dense_from, uint32_t *__restrict__ dense, uint32_t *__restrict__ control) {
    extern __shared__ __align__(16) uint8_t rv_raw[];
    float4 *xs = reinterpret_cast<float4 *>(rv_raw);
    float *lg = reinterpret_cast<float *>(rv_raw + (size_t)TB * hidden * 4); // [token][expert]
    uint32_t *items = reinterpret_cast<uint32_t *>(lg + TB * n_expert);        // expert << 16 | tokens
    uint32_t *mask = items + (TB + RV_TOKENS - 1) / RV_TOKENS * n_expert;    // by expert: the tokens it is left for
    __shared__ int n_items, n_left;
    __shared__ __align__(16) uint16_t cand[TB][32 + 64]; // by token: the experts left, up to 32, and room for their probabilities
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row4 = hidden / 4;
    const int t0 = blockIdx.x * TB, nt = min(TB, t - t0);
    if (tid == 0) n_items = n_left = 0;
    for (int e = tid; e < n_expert; e += RV_WARPS * 32) mask[e] = 0u;
    pdl_begin();
    for (int i = tid; i < nt * row4; i += RV_WARPS * 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s32(xs + i)), "l"(reinterpret_cast<const float4 *>(x + (size_t)t0 * hidden) + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    __syncthreads();
    int left = 0;      // experts left for the warp's token
    uint32_t mine = 0; // this lane's of them
    bool flat = false; // a row of zeros, of a padded prompt
    if (warp < nt) { // a warp's token: bounds of its scores
        const int tok = t0 + warp;
        float lo[PER], hi[PER], l[PER], W[PER], b[PER];
        bool finite = true, tiny = true;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int e = min(lane + 32 * j, n_expert - 1);
            l[j] = 0.f;
#pragma unroll
            for (int p = 0; p < RF_SPLITS; p++)
                if (p < splits) l[j] += approx[((size_t)p * t + tok) * n_expert + e];
            W[j] = wnorm[e] * 1.001f;
            b[j] = bias ? __ldg(bias + e) : 0.f;
        }
        float x2 = 0.f;
        for (int p = 0; p < splits; p++) x2 += xss[(size_t)p * t + tok];
        const float X = sqrtf(x2) * 1.001f, sub = 0x1p-25f * 1.01f * sqrtf((float)hidden);
        const float rel = 0x1p-10f + 0x1p-22f + 0x1p-18f + (float)hidden * (1.0625f * 0x1p-23f);
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const float d = X * W[j] * rel + sub * (X + W[j]);
            // the bias comes in by the addition of the specified score, which keeps the order whatever the bias is: an infinite one, which
            // excludes an expert or fixes it, and the type's lowest value bound the score as any other does
            lo[j] = __fadd_rn(route_bound(l[j] - d, -1.f), b[j]);
            hi[j] = __fadd_rn(route_bound(l[j] + d, 1.f), b[j]);
            finite = finite && isfinite(l[j]) && isfinite(d);
            tiny = tiny && X * W[j] < 0x1p-27f && W[j] < 1e8f;
        }
        // Logits below 2^-26 all have the sigmoid 0.5, exactly (1 + r rounds to 1 in its exponential), so none need be computed.  (Values whose squares
        // underflow are missing from X: 64 of 1.1e-19 times 1e8 are below 2^-27 as well.)
        flat = __all_sync(0xffffffffu, finite && tiny);
        const bool all = !__all_sync(0xffffffffu, finite);
        uint32_t key[PER], kth = 0u; // the top_k-th largest lower bound
#pragma unroll
        for (int j = 0; j < PER; j++) key[j] = lane + 32 * j < n_expert ? lmoe_score_key(lo[j]) : 0u;
        for (int k = 0; k < top_k; k++) {
            uint32_t best = 0u;
#pragma unroll
            for (int j = 0; j < PER; j++) best = max(best, key[j]);
            kth = __reduce_max_sync(0xffffffffu, best);
            bool take = lane == __ffs(__ballot_sync(0xffffffffu, best == kth)) - 1; // one of them is taken
#pragma unroll
            for (int j = 0; j < PER; j++) {
                const bool hit = take && key[j] == kth;
                key[j] = hit ? 0u : key[j];
                take = take && !hit;
            }
        }
#pragma unroll
        for (int j = 0; j < PER; j++) mine |= (uint32_t)(lane + 32 * j < n_expert && (all || lmoe_score_key(hi[j]) >= kth)) << j;
        left = flat ? 0 : (int)__reduce_add_sync(0xffffffffu, (uint32_t)__popc(mine));
        if (lane == 0) atomicAdd(&n_left, left);
    }
    __syncthreads();
    if (tid == 0) atomicAdd(control + LMOE_CONTROL_LEFT, (uint32_t)n_left);
    // where the bounds hardly tell the experts of a block's tokens apart, the tokens that keep too many go to route_dense_kernel
    const bool handed = left > dense_from && n_left > TB * dense_from + n_expert / 4;
    if (handed) {
        if (lane == 0) dense[atomicAdd(control + LMOE_CONTROL_DENSE, 1u)] = (uint32_t)(t0 + warp);
    } else if (flat) {
        for (int e = lane; e < n_expert; e += 32) lg[warp * n_expert + e] = 0.f;
    } else if (warp < nt) {
        int at = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int e = lane + 32 * j;
            const bool in = mine >> j & 1u;
            const uint32_t who = __ballot_sync(0xffffffffu, in);
            if (e < n_expert && !in) lg[warp * n_expert + e] = __uint_as_float(RV_OUT);
            if (in) {
                const int place = at + __popc(who & ((1u << lane) - 1u));
                if (place < 32) cand[warp][place] = (uint16_t)e;
                atomicOr(&mask[e], 1u << warp);
            }
            at += __popc(who);
        }
    }
    __syncthreads();
    for (int e = tid; e < n_expert; e += RV_WARPS * 32) {
        uint32_t m = mask[e];
        const int groups = (__popc(m) + RV_TOKENS - 1) / RV_TOKENS;
        if (!groups) continue;
        const int at = atomicAdd(&n_items, groups);
        for (int g = 0; g < groups; g++) {
            uint32_t part = 0u;
            for (int i = 0; i < RV_TOKENS && m; i++) {
                part |= m & (0u - m);
                m &= m - 1u;
            }
            items[at + g] = (uint32_t)e << 16 | part;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // A warp's items in turn, a router row in pieces of RV_PIECE passes: the next piece, this item's or the next one's first, is on its way while
    // one is multiplied.  The specified order: chains 4 lane .. 4 lane + 3, their elements in turn.
    const int n = n_items, steps = hidden / 128, pieces = (steps + RV_PIECE - 1) / RV_PIECE;
    if (warp < n) {
        float4 wa[RV_PIECE], wb[RV_PIECE];
        float acc[RV_TOKENS][4];
        int i = warp, piece = 0;
        uint32_t item = items[i];
        const float4 *w = reinterpret_cast<const float4 *>(router + (size_t)(item >> 16) * hidden) + lane;
        auto load = [&](float4 (&v)[RV_PIECE], const float4 *row, int p) {
#pragma unroll
            for (int u = 0; u < RV_PIECE; u++)
                if (p * RV_PIECE + u < steps) v[u] = __ldg(row + 32 * (p * RV_PIECE + u));
        };
        auto multiply = [&](const float4 (&v)[RV_PIECE], float4 (&after)[RV_PIECE]) { // false: that was the last piece
            const bool last = piece + 1 == pieces, more = i + RV_WARPS < n;
            const uint32_t now = item;
            const int p = piece;
            if (!last) {
                load(after, w, ++piece);
            } else if (more) {
                item = items[i += RV_WARPS];
                w = reinterpret_cast<const float4 *>(router + (size_t)(item >> 16) * hidden) + lane;
                load(after, w, piece = 0);
            }
            uint32_t m = now & 0xffffu;
#pragma unroll
            for (int c = 0; c < RV_TOKENS; c++) {
                if (m) {
                    const int tk = __ffs(m) - 1;
                    m &= m - 1u;
                    const float4 *xp = xs + tk * row4 + 32 * p * RV_PIECE + lane;
                    if (p == 0) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
#pragma unroll
                    for (int u = 0; u < RV_PIECE; u++)
                        if (p * RV_PIECE + u < steps) {
                            const float4 xv = xp[32 * u];
                            acc[c][0] = __fmaf_rn(xv.x, v[u].x, acc[c][0]);
                            acc[c][1] = __fmaf_rn(xv.y, v[u].y, acc[c][1]);
                            acc[c][2] = __fmaf_rn(xv.z, v[u].z, acc[c][2]);
                            acc[c][3] = __fmaf_rn(xv.w, v[u].w, acc[c][3]);
                        }
                    if (last) {
                        const float l = lmoe_router_fold(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
                        if (lane == 0) lg[tk * n_expert + (now >> 16)] = l;
                    }
                }
            }
            return !last || more;
        };
        load(wa, w, 0);
        while (multiply(wa, wb) && multiply(wb, wa)) {}
    }
    __syncthreads();
    if (warp >= nt || handed) return;
    uint32_t *ids_row = ids + (size_t)(t0 + warp) * top_k;
    float *w_row = weights + (size_t)(t0 + warp) * top_k, *probs = lg + warp * n_expert;
    if (!flat && left <= 32) {
        // a lane an expert: its slot is the number of those before it (a larger score, or the same and a lower index)
        const int e = lane < left ? cand[warp][lane] : 0;
        const float p = lane < left ? lmoe_sigmoid_fixed(probs[e]) : 0.f;
        const uint32_t key = lane < left ? lmoe_score_key(bias ? __fadd_rn(p, __ldg(bias + e)) : p) : 0u;
        int slot = 0;
        for (int i = 0; i < left; i++) { // (the list is in the order of the indices)
            const uint32_t other = __shfl_sync(0xffffffffu, key, i);
            slot += other > key || (other == key && i < lane);
        }
        const bool mine = lane < left && slot < top_k;
        float *by_slot = reinterpret_cast<float *>(cand[warp]) + 16; // behind the list: 32 floats
        if (mine) by_slot[slot] = p;
        __syncwarp();
        float w = p;
        if (norm) {
            float sum = 0.0f;
            for (int k = 0; k < top_k; k++) sum = __fadd_rn(sum, by_slot[k]);
            sum = sum < 6.103515625e-5f ? 6.103515625e-5f : sum;
            w = __fdiv_rn(w, sum);
        }
        if (scale != 0.0f && scale != 1.0f) w = __fmul_rn(w, scale);
        if (mine) {
            ids_row[slot] = (uint32_t)e;
            w_row[slot] = w;
        }
        return;
    }
    route_select_token<PER>(probs, bias, n_expert, top_k, scale, norm, ids_row, w_row, lane);
}

// The tokens that route_verify_kernel hands over: all their specified logits, as route_logits_tiled_kernel computes them, then the selection, by the block that
// finishes a tile's last share of the experts.  The number of tokens is known only here, so the tiles and shares are chosen here: by the
// time of the longest block, in half passes (of 16 tokens x 16 experts or 8 x 32; the staging of a tile is about a pass for 16 tokens).
template <int T, int PER>
__device__ __forceinline__ void route_dense(const float *router, const float *x, const float *bias, const uint32_t *list, int n, int passes, int hidden, int n_expert,
                                            int top_k, float scale, int norm, float *logits, uint32_t *done, uint32_t *ids, float *weights, uint8_t *smem) {
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, share = passes * (256 / T), shares = (n_expert + share - 1) / share;
    float *probs = reinterpret_cast<float *>(smem + (size_t)T * hidden * 4 + RT_FOLD) + warp * n_expert;
    for (int i = blockIdx.x; i < (n + T - 1) / T * shares; i += gridDim.x) {
        const int tile = i / shares, e0 = (i - tile * shares) * share, t0 = tile * T, nt = min(T, n - t0);
        route_tile<T>(router, [&](int k) { return x + (size_t)list[t0 + k] * hidden; }, nt, hidden, n_expert, e0, min(n_expert, e0 + share), smem,
                      logits + (size_t)t0 * n_expert);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            last = atomicAdd(done + tile, 1u) == (uint32_t)shares - 1u;
            __threadfence();
        }
        __syncthreads();
        if (last)
            for (int k = warp; k < nt; k += RT_THREADS / 32) {
                const size_t tok = list[t0 + k];
                for (int e = lane; e < n_expert; e += 32) probs[e] = __ldcg(logits + (size_t)(t0 + k) * n_expert + e);
                __syncwarp();
                route_select_token<PER>(probs, bias, n_expert, top_k, scale, norm, ids + tok * top_k, weights + tok * top_k, lane);
                __syncwarp();
            }
    }
}
template <int PER>
__global__ void __launch_bounds__(RT_THREADS, 1)
route_dense_kernel(const float *__restrict__ router, const float *__restrict__ x, const float *__restrict__ bias, const uint32_t *__restrict__ list,
                   const uint32_t *__restrict__ control, int hidden, int n_expert, int top_k, float scale, int norm, float *logits, uint32_t *done,
                   uint32_t *__restrict__ ids, float *__restrict__ weights, int sixteen) {
    extern __shared__ __align__(16) uint8_t rd_smem[];
    pdl_begin();
    const int n = (int)__ldcg(control + LMOE_CONTROL_DENSE);
    if (n == 0) return;
    // a lane a choice: 1 to 16 passes of 16 tokens, 1 to 8 of 8 (n_expert <= 256)
    const int lane = threadIdx.x & 31, g = (int)gridDim.x;
    auto cost = [&](int T, int p) {
        const int passes = (n_expert * T + 255) / 256, blocks = (n + T - 1) / T * ((passes + p - 1) / p);
        return p > passes || (T == 16 && !sixteen) ? 0xffffffffu : (uint32_t)((blocks + g - 1) / g * (2 * p + T / 8)) << 5;
    };
    const uint32_t mine = lane < 16 ? cost(16, 16 - lane) : (lane < 24 ? cost(8, 24 - lane) : 0xffffffffu);
    const int choice = (int)(__reduce_min_sync(0xffffffffu, mine == 0xffffffffu ? mine : mine | lane) & 31u);
    if (choice < 16) route_dense<16, PER>(router, x, bias, list, n, 16 - choice, hidden, n_expert, top_k, scale, norm, logits, done, ids, weights, rd_smem);
    else route_dense<8, PER>(router, x, bias, list, n, 24 - choice, hidden, n_expert, top_k, scale, norm, logits, done, ids, weights, rd_smem);
}

int rd_smem_bytes(int t, int64_t hidden, int64_t n_expert) { return (int)(t * hidden * 4 + RT_FOLD + RT_THREADS / 32 * n_expert * 4); }
int rv_smem(int tb, int64_t hidden, int64_t n_expert) { return (int)(tb * hidden * 4 + tb * n_expert * 4 + (tb + RV_TOKENS - 1) / RV_TOKENS * n_expert * 4 + n_expert * 4); }

} // namespace

// Whether the filter serves these sizes (hidden a whole number of the specified passes, experts a whole tile of the tensor core).
bool route_filter_available(int64_t hidden, int64_t n_expert, int64_t top_k) {
    return hidden % 128 == 0 && hidden >= 512 && hidden <= 4096 && n_expert % 32 == 0 && n_expert >= 64 && n_expert <= 256 && top_k <= 32 && top_k * 8 <= n_expert &&
           rv_smem(8, hidden, n_expert) <= 227 * 1024 - 4096;
}
// Scratch: the list of the tokens handed over and a count by tile of them, the router's f16 image, the norms, and the approximate logits by part of hidden, for at most this many token rows (never fewer for more
// tokens: a workspace for t tokens serves any smaller number).
static size_t rf_list_bytes(int64_t t) { return lmoe_align_up((size_t)t * 4, 256) + lmoe_align_up((size_t)(t + 7) / 8 * 4, 256); }
static int64_t rf_rows(int64_t t) { return t > 16384 ? t : (RF_SPLITS * t < 16384 ? RF_SPLITS * t : 16384); }
size_t route_filter_bytes(int64_t t, int64_t hidden, int64_t n_expert) {
    return rf_list_bytes(t) + lmoe_align_up((size_t)n_expert * hidden * 2, 256) + lmoe_align_up((size_t)n_expert * 4, 256) + lmoe_align_up((size_t)rf_rows(t) * 4, 256) +
           (size_t)rf_rows(t) * n_expert * 4;
}

cudaError_t launch_route_filter(const float *router, const float *bias, const float *x, int t, int hidden, int n_expert, int top_k, float scale, int norm,
                                void *scratch, uint32_t *ids, float *weights, uint32_t *flag, cudaStream_t s) {
    uint32_t *list = static_cast<uint32_t *>(scratch);
    uint32_t *done = list + lmoe_align_up((size_t)t * 4, 256) / 4;
    uint8_t *img = static_cast<uint8_t *>(scratch) + rf_list_bytes(t);
    float *wnorm = reinterpret_cast<float *>(img + lmoe_align_up((size_t)n_expert * hidden * 2, 256));
    float *xss = wnorm + lmoe_align_up((size_t)n_expert * 4, 256) / 4, *logits = xss + lmoe_align_up((size_t)rf_rows(t) * 4, 256) / 4;
    const int most = 227 * 1024 - 4096;
    static thread_local int c_dev = -1, c_sms = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev != c_dev) {
        if ((e = cudaDeviceGetAttribute(&c_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        for (auto f : {route_approx_kernel<128>, route_approx_kernel<64>})
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most - 1024)) != cudaSuccess) return e;
        for (auto f : {route_verify_kernel<16, 4>, route_verify_kernel<16, 8>, route_verify_kernel<8, 4>, route_verify_kernel<8, 8>})
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most)) != cudaSuccess) return e;
        for (auto f : {route_dense_kernel<4>, route_dense_kernel<8>})
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most)) != cudaSuccess) return e;
        c_dev = dev;
    }
    launch_pdl(route_prep_kernel, n_expert, 128, 0, s, router, hidden, n_expert, img, wnorm, flag, done, (t + 7) / 8);
    // 128 tokens a block where that covers two thirds of the device, else 64 and hidden in as many parts as there are SMs for
    const bool large = (t + 127) / 128 * 3 >= 2 * c_sms;
    const int tiles = large ? (t + 127) / 128 : (t + 63) / 64;
    int splits = 1;
    while (!large && splits < RF_SPLITS && tiles * splits * 2 <= c_sms && (int64_t)t * splits * 2 <= rf_rows(t) && hidden / 64 % (2 * splits) == 0) splits *= 2;
    launch_pdl(large ? route_approx_kernel<128> : route_approx_kernel<64>, dim3((unsigned)tiles, (unsigned)splits), 320,
               RF_STAGES * (RF_A_BYTES + n_expert * 128) + 1024, s, x, img, t, hidden, n_expert, logits, xss, flag);
    const bool dense = hidden % (128 * RT_AHEAD) == 0; // else a block computes what is left whatever it is, in no more time than the untiled product
    // sixteen tokens a block where the rows fit and the blocks are enough for the device
    const int tb = rv_smem(16, hidden, n_expert) <= most && (t + 15) / 16 * 5 >= 4 * c_sms ? 16 : 8;
    auto verify = n_expert <= 128 ? (tb == 16 ? route_verify_kernel<16, 4> : route_verify_kernel<8, 4>)
                                  : (tb == 16 ? route_verify_kernel<16, 8> : route_verify_kernel<8, 8>);
    launch_pdl(verify, (unsigned)((t + tb - 1) / tb), RV_WARPS * 32, rv_smem(tb, hidden, n_expert), s, router, x, bias, logits, xss, splits, wnorm, t, hidden,
               n_expert, top_k, scale, norm, ids, weights, dense ? n_expert / 4 : n_expert, list, flag);
    if (dense) {
        const bool sixteen = rd_smem_bytes(16, hidden, n_expert) <= most;
        launch_pdl(n_expert <= 128 ? route_dense_kernel<4> : route_dense_kernel<8>, (unsigned)c_sms, RT_THREADS,
                   rd_smem_bytes(sixteen ? 16 : 8, hidden, n_expert), s, router, x, bias, list, flag, hidden, n_expert, top_k, scale, norm, logits, done, ids,
                   weights, (int)sixteen);
    }
    return cudaGetLastError();
}
