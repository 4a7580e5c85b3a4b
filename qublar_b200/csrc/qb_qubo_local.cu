// Weighted QUBO sweep of a small problem: a CTA anneals 32 replicas, one per
// lane, with their fields and bit words in shared memory (up to about 860 bits).
//
// The lockstep sweep (qb_qubo.cu) closes every colour class with a grid
// barrier over the whole device; a small problem's classes hold a dozen bits,
// so nearly all of its time is that barrier (2.7 us a class step, 5 % issue).
// Here the warps of one CTA visit the bits, dealt to them in turn over all
// classes, and the barrier behind a class is joined by the warps of that class
// and the next only (named barriers in turn, as in qb_local.cu). A visit's row,
// couplings, own field and word and its draws do not depend on its neighbours'
// class: they are loaded and made for a warp's next bit as soon as it has
// finished one. Behind the barrier remain the neighbours' words, the walk of
// their flips and the decision.
//
// Bound: the dependent instructions of a visit in its warp. 120 bits of degree
// 12, 64 replicas x 1000 sweeps on a B200: 27 ms lockstep, 12.5 here (15 warps
// 16; 64 replicas to a warp with the lockstep sweep's transposed walk 21.8).
//
// Draws, arithmetic and visiting order are the lockstep sweep's, hence the
// branches too.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "qb_device.cuh"
#include "qb_internal.hpp"
#include "qb_philox.cuh"
#include "qb_qubo.hpp"
#include "qb_qubo_visit.cuh"

namespace qb {

namespace {

constexpr int kSmallMaxWarps = 24;
constexpr int kBarriers = 15;   // named barriers of the class steps
constexpr size_t kSmallSmem = size_t(224) * 1024;

struct QuboSmallArgs {
    int n;
    int n_colours;
    int sweeps;
    int refresh;
    int R;
    int warps;       // at most 15 x the smallest class: see the class barriers
    // 1: a visit's own field and word can be loaded as soon as the warp's visit
    // before it is done: the bit's last visit, n visits earlier, then lies in a
    // class before that one's (n >= widest class + warps)
    int ahead;
    uint64_t seed0;
    const int32_t* class_ptr;
    const int32_t* row;
    const int32_t* adj;
    const float* J;
    const float* h;
    const int32_t* order;
    const double* temp;
    uint8_t* x_out;
    float* drift;
    double* e_track;
    unsigned long long* accepts;
    double* trace;
};

__global__ void __launch_bounds__(32 * kSmallMaxWarps, 1) qubo_small_kernel(QuboSmallArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double s_tr[32];
    const int n = A.n, nc = A.n_colours, W = A.warps;
    uint2* xf = reinterpret_cast<uint2*>(smem);                    // (values, flips at the latest visit)
    float2* L = reinterpret_cast<float2*>(xf + n);                 // n x 32 fields (hi, lo)
    int32_t* cls = reinterpret_cast<int32_t*>(L + size_t(n) * 32);
    const int tid = int(threadIdx.x), lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0);
    // the CTA's first replica; replicas r and r + 32 of 64 share a draw block,
    // whose half this CTA takes
    const int b0 = int(blockIdx.x) * 32, half = int(blockIdx.x) & 1;
    const int R = min(32, A.R - b0);
    const bool has = lane < R;
    const uint64_t key = A.seed0 + uint64_t(b0 - 32 * half) + uint64_t(lane);
    for (int j = warp; j < n; j += W) {
        const float hj = A.h[j];
        L[size_t(j) * 32 + lane] = make_float2(hj, 0.0f);
        if (lane == 0) xf[j] = make_uint2(0u, 0u);
    }
    for (int c = tid; c <= nc; c += 32 * W) cls[c] = __ldg(A.class_ptr + c);
    if (tid < 32) s_tr[tid] = 0.0;
    __syncthreads();
    // bit j of sweep s is visit s n + j, made by warp (s n + j) mod W
    int j = warp, c0 = 0, s0 = 0;
    auto settle = [&]() {
        while (j >= n) {
            j -= n;
            ++s0;
            c0 = 0;
        }
        while (j >= cls[c0 + 1]) ++c0;
    };
    settle();
    // the visit in hand: loaded ahead of its class
    int k0 = 0, k1 = 0, nb = 0;
    float Jk = 0.0f;
    uint64_t u53 = 0;
    float2 own{};
    uint32_t xj = 0;
    auto load_state = [&]() {
        own = L[size_t(j) * 32 + lane];
        xj = xf[j].x;
    };
    auto issue = [&]() {
        k0 = __ldg(A.row + j);
        k1 = __ldg(A.row + j + 1);
        u53 = draw_u53_half(key, uint32_t(__ldg(A.order + j)), uint32_t(s0), 0u, half);
        nb = 0;
        Jk = 0.0f;
        if (k0 + lane < k1) {
            nb = __ldg(A.adj + k0 + lane);
            Jk = __ldg(A.J + k0 + lane);
        }
        if (A.ahead) load_state();
    };
    issue();
    auto members = [&](int c) {
        const int d = c + 1 < nc ? c + 1 : 0;
        return 32 * min(W, cls[c + 1] - cls[c] + cls[d + 1] - cls[d]);
    };
    auto wait_class = [&](int idx, int threads) {
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(1 + idx % kBarriers), "r"(threads) : "memory");
    };
    auto leave_class = [&](int idx, int threads) {
        __syncwarp();
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + idx % kBarriers), "r"(threads) : "memory");
    };
    auto full_stop = [&](int sweep) { return sweep > 0 && A.trace != nullptr; };
    bool ready = s0 == 0 && c0 == 0;
    float eh = 0.0f, el = 0.0f, drift = 0.0f;
    unsigned long long accepts = 0;
    int turn = 0;   // sweep x classes modulo kBarriers
    for (int sweep = 0; sweep < A.sweeps; ++sweep, turn = (turn + nc) % kBarriers) {
        if (full_stop(sweep)) {
            __syncthreads();
            if (tid < R) {
                A.trace[size_t(b0 + tid) * A.sweeps + sweep - 1] = s_tr[tid];
                s_tr[tid] = 0.0;
            }
            __syncthreads();
        }
        const double T = A.temp[sweep];
        const float inv_T = float(1.0 / T);
        const bool refresh = A.refresh > 0 && sweep > 0 && sweep % A.refresh == 0;
        while (s0 == sweep) {
            const int c = c0, idx = turn + c;   // the barrier behind class c, modulo kBarriers
            if (!ready && !(c == 0 && full_stop(sweep))) wait_class(idx + kBarriers - 1, members(c > 0 ? c - 1 : nc - 1));
            do {
                if (!A.ahead) load_state();
                float hi = own.x, lo = own.y;
                double full = refresh ? double(__ldg(A.h + j)) : 0.0;
                for (int kb = k0; kb < k1; kb += 32) {
                    const bool live = kb + lane < k1;
                    if (kb > k0) {   // a row of more than 32 neighbours
                        nb = live ? __ldg(A.adj + kb + lane) : 0;
                        Jk = live ? __ldg(A.J + kb + lane) : 0.0f;
                    }
                    uint2 w = make_uint2(0u, 0u);
                    if (live) w = xf[nb];
                    // the neighbours that some replica flipped (all of them in a
                    // refresh sweep, whose sum needs every value), in CSR order, four
                    // at a time; a zero delta leaves a replica's field as it is
                    unsigned todo = __ballot_sync(kFullMask, refresh ? live : w.y != 0u);
                    while (todo) {
                        float Jq[4];
                        uint32_t xq[4], fq[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int q = todo ? __ffs(todo) - 1 : 0;
                            const bool some = todo != 0;
                            todo &= todo - 1u;
                            Jq[u] = __shfl_sync(kFullMask, Jk, q);
                            xq[u] = some ? __shfl_sync(kFullMask, w.x, q) : 0u;
                            fq[u] = some ? __shfl_sync(kFullMask, w.y, q) : 0u;
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const bool on = (xq[u] >> lane) & 1u;
                            two_sum_acc(hi, lo, (fq[u] >> lane) & 1u ? (on ? Jq[u] : -Jq[u]) : 0.0f);
                            if (refresh && on) full += double(Jq[u]);
                        }
                    }
                }
                if (refresh) {
                    if (has) drift = fmaxf(drift, float(fabs(double(__fadd_rn(hi, lo)) - full)));
                    hi = float(full);
                    lo = float(full - double(hi));
                }
                const float field = __fadd_rn(hi, lo);
                const float dE = (xj >> lane) & 1u ? -field : field;
                const bool acc = has && (dE <= 0.0f || uphill_accept(u53, double(dE), T, inv_T));   // NaN: rejected
                const unsigned mask = __ballot_sync(kFullMask, acc);
                if (lane == 0) xf[j] = make_uint2(xj ^ mask, mask);
                if (acc) {
                    two_sum_acc(eh, el, dE);
                    ++accepts;
                    if (A.trace) atomicAdd(&s_tr[lane], double(dE));
                }
                L[size_t(j) * 32 + lane] = make_float2(hi, lo);
                __syncwarp();
                j += W;
                settle();
                if (s0 < A.sweeps) issue();
            } while (s0 == sweep && c0 == c);
            const bool last = c == nc - 1;
            if (last && (sweep + 1 == A.sweeps || full_stop(sweep + 1))) {
                ready = false;
            } else if (last ? s0 == sweep + 1 && c0 == 0 : s0 == sweep && c0 == c + 1) {
                wait_class(idx, members(c));
                ready = true;
            } else {
                leave_class(idx, members(c));
                ready = false;
            }
        }
    }
    __syncthreads();
    if (A.trace && tid < R) A.trace[size_t(b0 + tid) * A.sweeps + A.sweeps - 1] = s_tr[tid];
    if (has)
        for (int i = warp; i < n; i += W)
            A.x_out[size_t(b0 + lane) * size_t(n) + size_t(__ldg(A.order + i))] = uint8_t((xf[i].x >> lane) & 1u);
    if (has) {
        if (drift > 0.0f) atomicMax(reinterpret_cast<int*>(&A.drift[b0 + lane]), __float_as_int(drift));
        if (accepts) atomicAdd(&A.accepts[b0 + lane], accepts);
        atomicAdd(&A.e_track[b0 + lane], double(eh) + double(el));
    }
}

struct ClassSizes {
    int smallest, widest;
};
ClassSizes class_sizes(const QuboPlan& p) {
    ClassSizes s{p.n, 0};
    for (int c = 0; c < p.col.n_colours(); ++c) {
        const int k = p.col.class_ptr[size_t(c) + 1] - p.col.class_ptr[size_t(c)];
        s.smallest = std::min(s.smallest, k);
        s.widest = std::max(s.widest, k);
    }
    return s;
}

size_t small_smem(const QuboPlan& p) { return size_t(p.n) * (32 * 8 + 8) + (size_t(p.col.n_colours()) + 1) * 4; }

}  // namespace

// A class step costs about 1.3 us per round of the CTA's warps, the cooperative
// sweep's 3.5 to 5 us: up to two rounds of an average class (120 bits of degree
// 12, 300 sweeps: 3.9 against 8.2 ms; 400 bits in 5 classes of 80: 9.4 against 6.7).
bool qubo_small_fit(const QuboPlan& p) {
    const char* k = std::getenv("QB_QUBO_KERNEL");   // "lockstep" and "small" ask for one of the two
    if (small_smem(p) > kSmallSmem || (k && *k == 'l')) return false;
    return (k && *k == 's') || p.n <= 2 * kSmallMaxWarps * p.col.n_colours();
}

qb_status launch_qubo_small(const QuboPlan& p, const QuboBuffers& b, int R, int sweeps, int refresh, uint64_t seed0,
                            cudaStream_t st) {
    QuboSmallArgs A{};
    A.n = p.n;
    A.n_colours = p.col.n_colours();
    A.sweeps = sweeps;
    A.refresh = refresh;
    A.R = R;
    A.seed0 = seed0;
    const ClassSizes cs = class_sizes(p);
    // a barrier's name comes round after 15 classes: with W warps and at least
    // W / 15 bits in every class, a warp's next bit lies at most 15 classes ahead
    A.warps = std::max(1, std::min({kSmallMaxWarps, kBarriers * cs.smallest, 2 * cs.widest}));
    A.ahead = p.n >= cs.widest + A.warps ? 1 : 0;
    A.class_ptr = p.d_class_ptr.as<int32_t>();
    A.row = p.d_row.as<int32_t>();
    A.adj = p.d_adj.as<int32_t>();
    A.J = p.d_J.as<float>();
    A.h = p.d_h.as<float>();
    A.order = p.d_order.as<int32_t>();
    A.temp = b.temp;
    A.x_out = b.x;
    A.drift = b.drift;
    A.e_track = b.e_track;
    A.accepts = b.accepts;
    A.trace = b.trace;
    QB_CUDA(allow_max_smem(qubo_small_kernel));
    qubo_small_kernel<<<unsigned((R + 31) / 32), 32 * A.warps, small_smem(p), st>>>(A);
    QB_CUDA(cudaGetLastError());
    count_sweep(Sweep::kQuboSmall);
    return QB_OK;
}

}  // namespace qb
