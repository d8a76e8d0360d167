// The f32 router product of a tile of tokens, in the specified order (route_math.cuh): what route.cu and route_filter.cu share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace {

// hidden a multiple of 512: a register-tiled product over the 128 partial chains of the specified order.
// A block stages up to T tokens in shared memory and walks its share of the experts.  Four sets of two warps serve eight tokens by
// eight experts each; lane l of warp w of a set owns the chains 64w + 2l and 64w + 2l + 1, and a thread multiplies the eight
// tokens by the eight experts for those two: one fma.rn.f32x2 each (two independent IEEE fmas, so the logits are
// bit-identical).  Two things bound such a product: the operand words a lane takes in per fma, as shared memory and L1 hand out
// 32 of them a cycle however many lanes ask for the same, and the instructions beside the fmas, which leave every second issue
// slot.  8 x 8 x 2 chains take 32 words and 20 other instructions for 64 double fmas; 8 x 4 x 4 took 48 words, 16 x 8 x 1
// only 24, but 90 instructions (with the selection, 16384 tokens x 256 experts x 3072: 809 and 869 us, this 692; 2048 tokens:
// 120, 127, 104).  The router words come straight from L2 into registers, RT_AHEAD steps ahead.
// The fold of a (token, expert) pair is the specified one: the four chains of a lane pair, then stride 16 across the two warps
// (through shared memory) and 8, 4, 2, 1 across the lane pairs; a step keeps half of the values.
constexpr int RT_THREADS = 256;
constexpr int RT_AHEAD = 4;
constexpr int RT_FOLD = 4 * 2 * 4 * 32 * 16; // bytes of the four sets' fold buffers

__device__ __forceinline__ void fma_f32x2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// x_row(i): token i's row, i < nt; experts e0 to e_end; logits of the tile's first token, in global or shared memory.  The experts' words are
// asked for before the tokens' are waited for; smem (T * hidden * 4 + RT_FOLD bytes) is free again after a barrier.
template <int T, typename Row>
__device__ __forceinline__ void route_tile(const float *__restrict__ router, Row x_row, int nt, int hidden, int n_expert, int e0, int e_end, uint8_t *rt_smem,
                                           float *__restrict__ logits) {
    constexpr int TG = T / 8, EG = 4 / TG; // token and expert groups of the four sets
    typedef unsigned long long u64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = warp & 1, set = warp >> 1, tg = set % TG, eg = set / TG;
    const int steps = hidden / 128;
    float4 *fold = reinterpret_cast<float4 *>(rt_smem + (size_t)T * hidden * 4) + set * (2 * 4 * 32);
    // staged as [step][token][chain]; tokens past the last one hold whatever was there, their results are not written
    for (int i = threadIdx.x; i < nt * (hidden / 4); i += RT_THREADS) {
        const int tok = i / (hidden / 4), c = i - tok * (hidden / 4);
        cp_async16(rt_smem + ((size_t)(c / 32) * T + tok) * 512 + c % 32 * 16, reinterpret_cast<const float4 *>(x_row(tok)) + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // this thread's word of its router rows, RT_AHEAD steps on (rows past the last one repeat it)
    const u64 *rp[8];
    auto rows = [&](int e1) {
#pragma unroll
        for (int e = 0; e < 8; e++)
            rp[e] = reinterpret_cast<const u64 *>(router + (size_t)min(e1 + 8 * eg + e, n_expert - 1) * hidden) + 32 * w + lane;
    };
    rows(e0);
    u64 wq[RT_AHEAD][8];
#pragma unroll
    for (int u = 0; u < RT_AHEAD; u++)
#pragma unroll
        for (int e = 0; e < 8; e++) wq[u][e] = __ldg(rp[e] + 64 * u);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (; e0 < e_end; e0 += 8 * EG) {
        u64 acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) acc[i][e] = 0ull;
        const u64 *xp = reinterpret_cast<const u64 *>(rt_smem) + tg * 8 * 64 + 32 * w + lane;
        // steps is a multiple of RT_AHEAD (the launcher sees to it)
#pragma unroll 1
        for (int j = 0; j < steps; j += RT_AHEAD) {
            if (j + RT_AHEAD == steps) rows(e0 + 8 * EG); // the words of the next pass
            else
#pragma unroll
                for (int e = 0; e < 8; e++) rp[e] += 64 * RT_AHEAD;
#pragma unroll
            for (int u = 0; u < RT_AHEAD; u++) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const u64 xv = xp[i * 64];
#pragma unroll
                    for (int e = 0; e < 8; e++) fma_f32x2(acc[i][e], xv, wq[u][e]);
                }
                xp += T * 64;
#pragma unroll
                for (int e = 0; e < 8; e++) wq[u][e] = __ldg(rp[e] + 64 * u);
            }
        }
        auto halve = [&](float lo, float hi, int st) { // the lane keeps lo or hi by that bit of it
            const bool up = (lane & st) != 0;
            return __fadd_rn(up ? hi : lo, __shfl_xor_sync(0xffffffffu, up ? lo : hi, st));
        };
        // chains 4 L .. 4 L + 3: (first + second) + (third + fourth); value 8 e + i of the four experts kept
        float v[32];
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float2 lo = *reinterpret_cast<const float2 *>(&acc[i][e]), hi = *reinterpret_cast<const float2 *>(&acc[i][e + 4]);
                v[8 * e + i] = halve(__fadd_rn(lo.x, lo.y), __fadd_rn(hi.x, hi.y), 1);
            }
        // across the two warps: each hands over the half that the other finishes
        float r[16];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const float4 lo = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
            const float4 hi = make_float4(v[16 + 4 * h], v[17 + 4 * h], v[18 + 4 * h], v[19 + 4 * h]);
            fold[(w * 4 + h) * 32 + lane] = w ? lo : hi;
            r[4 * h] = w ? hi.x : lo.x; r[4 * h + 1] = w ? hi.y : lo.y; r[4 * h + 2] = w ? hi.z : lo.z; r[4 * h + 3] = w ? hi.w : lo.w;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + set) : "memory");
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const float4 o = fold[((w ^ 1) * 4 + h) * 32 + lane];
            r[4 * h] = __fadd_rn(r[4 * h], o.x); r[4 * h + 1] = __fadd_rn(r[4 * h + 1], o.y);
            r[4 * h + 2] = __fadd_rn(r[4 * h + 2], o.z); r[4 * h + 3] = __fadd_rn(r[4 * h + 3], o.w);
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + set) : "memory"); // the buffer is free for the next pass
#pragma unroll
        for (int i = 0; i < 8; i++) r[i] = halve(r[i], r[i + 8], 16);
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = halve(r[i], r[i + 4], 8);
#pragma unroll
        for (int i = 0; i < 2; i++) r[i] = halve(r[i], r[i + 2], 4);
        r[0] = halve(r[0], r[1], 2);
        // value 16 w + (bits 4, 3, 2, 1 of the lane): expert half by bit 0, expert by the upper two bits, token by the lower three
        const int val = 16 * w + ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
        const int tok = 8 * tg + val % 8, ex = e0 + 8 * eg + (lane & 1) * 4 + val / 8;
        if (tok < nt && ex < e_end) logits[(size_t)tok * n_expert + ex] = r[0];
    }
}

} // namespace
