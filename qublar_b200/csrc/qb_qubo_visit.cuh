// Device code of a weighted-QUBO visit. Both sweeps (qb_qubo.cu,
// qb_qubo_local.cu) add flips by two_sum_acc; the walk over the flipped
// neighbours is the cooperative sweep's: a warp visits one bit for 64 replicas,
// lane l serves replicas l and l + 32 (the small sweep, 32 replicas to a warp,
// adds every flipped neighbour to all of them, masked).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace qb {

constexpr unsigned kFullMask = 0xffffffffu;

// 32 x 32 bit transpose across the warp: lane p returns the word whose bit q
// is bit p of lane q's w (five rounds of block swaps between lanes l, l ^ j).
__device__ __forceinline__ unsigned warp_transpose32(unsigned w, int lane) {
#pragma unroll
    for (int j = 16; j >= 1; j >>= 1) {
        const unsigned L = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u
                                                                          : 0x55555555u;
        const unsigned o = __shfl_xor_sync(kFullMask, w, j);
        w = (lane & j) ? ((w & ~L) | ((o & ~L) >> j)) : ((w & L) | ((o & L) << j));
    }
    return w;
}

// hi + lo += v, the rounding error of the fp32 add carried into lo (Knuth's
// TwoSum; no fused operations).
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float v) {
    const float s = __fadd_rn(hi, v);
    const float bp = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(v, bp));
    hi = s;
    lo = __fadd_rn(lo, e);
}

// One batch of up to 32 neighbours (lane q holds neighbour q's coupling Jk,
// value word x and flip word f): the deltas of the flips added to the fields.
__device__ __forceinline__ void apply_flips(int lane, float Jk, unsigned long long f, unsigned long long x, float& hi0,
                    float& lo0, float& hi1, float& lo1) {
    // each lane walks, in CSR order, the neighbours that one of its two
    // replicas flipped: bit q of F0 (F1) = neighbour kb + q flipped in
    // replica r0 (r1), so the warp iterates over the busiest lane's
    // flips instead of every neighbour that any replica flipped
    if (__ballot_sync(kFullMask, f != 0ull) == 0u) return;
    const unsigned F0 = warp_transpose32(uint32_t(f), lane);
    const unsigned F1 = warp_transpose32(uint32_t(f >> 32), lane);
    const unsigned xlo = uint32_t(x), xhi = uint32_t(x >> 32);
    // each replica walks its own flipped neighbours (ascending: CSR
    // order), two steps of both lists per iteration, so the warp runs
    // max(flips of r0, flips of r1) of its busiest lane, not their union
    unsigned t0 = F0, t1 = F1;
    while (__any_sync(kFullMask, (t0 | t1) != 0u)) {
        unsigned b0[2], b1[2];
        float J0[2], J1[2];
        unsigned xl[2], xh[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            b0[u] = t0 & (0u - t0);
            t0 ^= b0[u];
            b1[u] = t1 & (0u - t1);
            t1 ^= b1[u];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q0 = b0[u] ? __ffs(b0[u]) - 1 : 0, q1 = b1[u] ? __ffs(b1[u]) - 1 : 0;
            J0[u] = __shfl_sync(kFullMask, Jk, q0);
            J1[u] = __shfl_sync(kFullMask, Jk, q1);
            xl[u] = __shfl_sync(kFullMask, xlo, q0);
            xh[u] = __shfl_sync(kFullMask, xhi, q1);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (b0[u]) two_sum_acc(hi0, lo0, ((xl[u] >> lane) & 1u) ? J0[u] : -J0[u]);
            if (b1[u]) two_sum_acc(hi1, lo1, ((xh[u] >> lane) & 1u) ? J1[u] : -J1[u]);
        }
    }
}

// The same in a refresh sweep: every live neighbour is walked in CSR order (the
// fp64 sums a0, a1 need every x).
__device__ __forceinline__ void apply_flips_refresh(int lane, bool live, float Jk, unsigned long long f, unsigned long long x,
                            float& hi0, float& lo0, float& hi1, float& lo1, double& a0, double& a1) {
    const int r0 = lane, r1 = lane + 32;
    unsigned todo = __ballot_sync(kFullMask, live);
    while (todo) {
        const int q = __ffs(todo) - 1;
        todo &= todo - 1u;
        const unsigned long long fq = __shfl_sync(kFullMask, f, q);
        const unsigned long long xq = __shfl_sync(kFullMask, x, q);
        const float Jq = __shfl_sync(kFullMask, Jk, q);
        if ((fq >> r0) & 1ull) two_sum_acc(hi0, lo0, ((xq >> r0) & 1ull) ? Jq : -Jq);
        if ((fq >> r1) & 1ull) two_sum_acc(hi1, lo1, ((xq >> r1) & 1ull) ? Jq : -Jq);
        if ((xq >> r0) & 1ull) a0 += double(Jq);
        if ((xq >> r1) & 1ull) a1 += double(Jq);
    }
}

}  // namespace qb
