// Residual sweep with a CTA per branch: the branch's residual pairs and bits
// live in the CTA's shared memory (up to about 27,000 rays).
//
// The lockstep sweep (qb_kernels.cu) keeps all branches in global memory and
// closes every colour class with a grid barrier: about 4 us a class step
// whatever the class holds. Branches do not interact, so a branch that fits one
// SM needs no grid at all: a class step is gathers from shared memory and a
// barrier of the warps that take part.
//
// A warp item is 16 lane pairs, a pair per 16-entry segment of a bit (the even
// and the odd entries' fmaf chains, as in the lockstep sweep), a bit's pairs
// side by side: its segment sums are added in order through shuffles, every
// lane of the bit takes the decision, and each lane updates the residuals it
// holds -- no block barrier inside a class. A bit of more than 16 segments
// takes a warp to itself and goes over its segments in rounds. What does not
// depend on the state (record, entries, neighbour list, draw) is loaded and
// computed for a warp's next item as soon as it has finished one; items are
// dealt to the warps in a row over all classes, so that is a class or more
// ahead of its use.
//
// Bound: the dependent instructions of an item in its warp (about 1 us a class
// step; loads and draws are off it), on larger problems the items per SM.
// Measured on a B200, 100 sweeps: 5,020 bits, 24 branches 34.9 ms lockstep,
// 10.2 here (12.9 with the next item's loads ahead of a CTA-wide barrier, 11.6
// with items dealt in turn, 10.2 with barriers of the two classes' warps only);
// 20,000 bits, 16 branches 52 and 31; 40,000 bits, 64 branches 83 and 54.
//
// The arithmetic, the draws and hence the branches are the lockstep sweep's.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "qb_device.cuh"
#include "qb_local.hpp"
#include "qb_philox.cuh"

namespace qb {

namespace {

constexpr unsigned kAllLanes = 0xffffffffu;
constexpr int kLocalThreads = 480;   // 15 warps: see the class barriers
constexpr int kLocalWarps = kLocalThreads / 32;
constexpr int kPairs = 16;          // segments per warp item
constexpr int kSegE = 16;           // entries per segment
constexpr int kHold = kSegE / 2;    // entries per lane
constexpr int kNbrLane = 3;         // neighbours per lane loaded ahead (two lanes of a bit share them)
constexpr size_t kLocalSmem = size_t(224) * 1024;
constexpr uint32_t kRay = 0x7FFFFFFFu;   // entry word 0: ray | (w < 0) << 31

struct ResidLocalArgs {
    int n;
    int n_rays;
    int n_colours;
    int sweeps;
    int refresh;
    float lambda;
    uint64_t seed0;
    const uint4* rec;          // per lane pair 2 x uint4 (see resid_local_plan)
    const int32_t* item_ptr;   // n_colours + 1: warp items of each class
    const uint2* ent;
    const int32_t* nbr;        // sweep positions
    const int32_t* order;
    const double* d;
    const double* w64;
    const int32_t* rrow;
    const int32_t* rbit;       // sweep position of each ray-major entry
    const float* ra;
    const double* temp;
    uint8_t* x_out;
    float* drift;
    unsigned long long* accepts;
    double* trace;
};

// A lane pair's record: first entry of its segment; segment length | first pair
// of its bit << 5 | length of the bit's last segment << 10 | the bit's segments
// << 16 (0: empty pair); the bit's sweep position; its input index; lin, q,
// first neighbour, neighbours.
// The cluster order's record: first entry; rays | flags; the rest alike.
constexpr uint32_t kHeavyTag = 1u << 16, kLiveTag = 1u << 17;
constexpr int kGroupRecs = 4;
constexpr int kHeavyRays = 64;
__host__ __device__ inline uint32_t rec_tag(int len, int pair, int last, int segs) {
    return uint32_t(len) | uint32_t(pair) << 5 | uint32_t(last) << 10 | uint32_t(segs) << 16;
}

// GROUPS: the cluster sweep's order (qb_kernels.cu) instead: eight lanes per
// bit, 32 for one of more than 64 rays, each the fmaf chain over every eighth
// (32nd) entry, joined by an xor butterfly; an item is four bits or one heavy
// bit, and a lane past its eight entries goes on with the same chain.
template <bool GROUPS>
__global__ void __launch_bounds__(kLocalThreads, 1) resid_local_kernel(ResidLocalArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double s_trace;
    __shared__ unsigned long long s_accepts;
    const int nr = A.n_rays, n = A.n, nc = A.n_colours, words = (n + 31) / 32;
    float2* rho = reinterpret_cast<float2*>(smem);
    uint32_t* xs = reinterpret_cast<uint32_t*>(rho + nr + 1);
    int32_t* ip = reinterpret_cast<int32_t*>(xs + words);
    const int tid = int(threadIdx.x), lane = tid & 31;
    const int warp = __shfl_sync(kAllLanes, tid >> 5, 0);
    const int pair = GROUPS ? lane >> 3 : lane >> 1, half = lane & 1;
    constexpr int kRecs = GROUPS ? kGroupRecs : kPairs;   // records per item
    const int branch = int(blockIdx.x);
    const uint64_t seed = A.seed0 + uint64_t(branch);
    for (int b = tid; b < nr; b += kLocalThreads) rho[b] = split_pair(-__dmul_rn(sqrt(fabs(A.w64[b])), A.d[b]));
    for (int k = tid; k < words; k += kLocalThreads) xs[k] = 0u;
    if (tid == 0) rho[nr] = make_float2(0.0f, 0.0f);
    for (int c = tid; c <= nc; c += kLocalThreads) ip[c] = __ldg(A.item_ptr + c);
    if (tid == 0) {
        s_trace = 0.0;
        s_accepts = 0;
    }
    __syncthreads();

    auto bit_of = [&](int i) { return (xs[i >> 5] >> (i & 31)) & 1u; };
    // The items of all classes in a row are dealt to the warps in turn, so a
    // warp's next item lies a class or more ahead and its loads and draw run
    // while other warps have the current class.
    const int total = ip[nc];
    int c0 = 0, it0 = warp, s0 = 0;
    auto settle = [&]() {   // the class of item it0 (of a later sweep past the end)
        while (it0 >= total) {
            it0 -= total;
            ++s0;
            c0 = 0;
        }
        while (it0 >= ip[c0 + 1]) ++c0;
    };
    auto rec_of = [&](int it) { return A.rec + (size_t(it) * kRecs + size_t(pair)) * 2; };
    // The item in hand: its record, and per entry of the lane its residual and
    // coefficient; entries past the segment are the zero pair rho[nr] with a
    // zero coefficient, which change nothing. na, nb: the next item's record.
    // issue() starts the loads and makes the draw, nothing in it waits for
    // them: it runs ahead of the barrier, whose wait hides them for every warp
    // but the class's last, whose arrival comes behind it.
    uint4 ra{}, rb{}, na{}, nb{};
    uint2 en[kHold];
    int nbr[kNbrLane];
    uint64_t u53 = 0;
    auto issue = [&]() {
        ra = na;
        rb = nb;
        int ni = it0 + kLocalWarps;
        while (ni >= total) ni -= total;
        const uint4* next = rec_of(ni);
        na = __ldg(next);
        nb = __ldg(next + 1);
        if constexpr (GROUPS) {
            const int rays = int(ra.y & 0xFFFFu);
            const bool heavy = (ra.y & kHeavyTag) != 0;
            const int gl = heavy ? lane : lane & 7, G = heavy ? 32 : 8;
#pragma unroll
            for (int u = 0; u < kHold; ++u) {
                en[u] = make_uint2(uint32_t(nr), 0u);
                if (gl + G * u < rays) en[u] = __ldg(A.ent + ra.x + gl + G * u);
            }
            nbr[0] = gl < int(rb.w) && (ra.y & kLiveTag) ? __ldg(A.nbr + rb.z + gl) : -1;
        } else {
            const int len = int(ra.y & 31u);
#pragma unroll
            for (int u = 0; u < kHold; ++u) {
                en[u] = make_uint2(uint32_t(nr), 0u);
                if (half + 2 * u < len) en[u] = __ldg(A.ent + ra.x + half + 2 * u);
            }
            // lanes 0 and 1 of the bit share its neighbours
            const int gl = lane - 2 * int((ra.y >> 5) & 31u);
#pragma unroll
            for (int t = 0; t < kNbrLane; ++t)
                nbr[t] = (ra.y >> 16) && gl < 2 && gl + 2 * t < int(rb.w) ? __ldg(A.nbr + rb.z + gl + 2 * t) : -1;
        }
        u53 = draw_u53(seed, ra.w, uint32_t(s0), 0u);
    };
    auto coef = [](const uint2& e) { return (e.x >> 31) ? -__uint_as_float(e.y) : __uint_as_float(e.y); };
    if (total > 0) {
        settle();
        na = __ldg(rec_of(it0));
        nb = __ldg(rec_of(it0) + 1);
        issue();
    }
    // The barrier between a class and the next is joined by the warps that have
    // items in either: those of the first only arrive, those of the second wait
    // (named barriers 1 .. 15 in turn). A barrier's name comes round after 15
    // classes: every class has an item, so with 15 warps a warp's next item lies
    // at most 15 classes ahead, and when it comes to wait at the barrier before
    // that class (at most 14 after the one it last joined), the last use of the
    // name has completed. A refresh or a trace stops the whole CTA instead.
    auto full_stop = [&](int sweep) {   // before the sweep's first class
        return sweep > 0 && (A.trace != nullptr || (A.refresh > 0 && sweep % A.refresh == 0));
    };
    auto members = [&](int c) {   // threads of the barrier behind class c
        const int d = c + 1 < nc ? c + 1 : 0;
        return 32 * min(kLocalWarps, ip[c + 1] - ip[c] + ip[d + 1] - ip[d]);
    };
    auto wait_class = [&](int idx, int threads) {
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(1 + idx % 15), "r"(threads) : "memory");
    };
    auto leave_class = [&](int idx, int threads) {
        __syncwarp();
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + idx % 15), "r"(threads) : "memory");
    };
    bool ready = s0 == 0 && c0 == 0;   // nothing to wait for before the item in hand
    unsigned long long my_accepts = 0;
    int turn = 0;   // sweep x classes modulo 15
    for (int sweep = 0; sweep < A.sweeps; ++sweep, turn = (turn + nc) % 15) {
        if (full_stop(sweep)) {
            __syncthreads();
            if (A.trace && tid == 0) {   // the sweep before
                A.trace[size_t(branch) * A.sweeps + sweep - 1] = s_trace;
                s_trace = 0.0;
            }
            if (A.refresh > 0 && sweep % A.refresh == 0) {
                // fp64 refresh, a thread per ray: rho = sum a' over its set bits in
                // order - sqrt|w| d, the drift |hi + lo - rho| recorded
                float dmax = 0.0f;
                for (int b = tid; b < nr; b += kLocalThreads) {
                    const double sw = sqrt(fabs(A.w64[b]));
                    double acc = 0.0;
                    const int k1 = A.rrow[b + 1];
                    for (int k = A.rrow[b]; k < k1; ++k)
                        if (bit_of(__ldg(A.rbit + k))) acc = __dadd_rn(acc, double(scaled_coef(sw, __ldg(A.ra + k))));
                    const double v = __dsub_rn(acc, __dmul_rn(sw, A.d[b]));
                    const float2 r = rho[b];
                    dmax = fmaxf(dmax, __double2float_rn(fabs(__dsub_rn(__dadd_rn(double(r.x), double(r.y)), v))));
                    rho[b] = split_pair(v);
                }
                if (dmax > 0.0f) atomicMax(reinterpret_cast<int*>(&A.drift[branch]), __float_as_int(dmax));
            }
            __syncthreads();
        }
        const double T = A.temp[sweep];
        const float inv_T = float(1.0 / T);
        while (s0 == sweep && total > 0) {
            const int c = c0, idx = turn + c;   // the barrier behind class c, modulo 15
            if (!ready && !(c == 0 && full_stop(sweep))) wait_class(idx + 15 - 1, members(c > 0 ? c - 1 : nc - 1));
            do {   // the warp's items of this class
                if constexpr (GROUPS) {
                    const bool heavy = (ra.y & kHeavyTag) != 0, live = (ra.y & kLiveTag) != 0;   // heavy: warp-uniform
                    const int gl = heavy ? lane : lane & 7, G = heavy ? 32 : 8;
                    const int rays = int(ra.y & 0xFFFFu), i = int(ra.z);
                    float2 held[kHold];
#pragma unroll
                    for (int u = 0; u < kHold; ++u) held[u] = rho[en[u].x & kRay];
                    const uint32_t xi = bit_of(i);
                    int unlike = nbr[0] >= 0 ? int(bit_of(nbr[0]) ^ xi) : 0;
                    if (live)
                        for (int q = gl + G; q < int(rb.w); q += G) unlike += int(bit_of(__ldg(A.nbr + rb.z + q)) ^ xi);
                    float acc = 0.0f;
#pragma unroll
                    for (int u = 0; u < kHold; ++u) acc = fmaf(coef(en[u]), __fadd_rn(held[u].x, held[u].y), acc);
                    for (int e = gl + G * kHold; e < rays; e += G) {   // a heavy bit of more than 256 rays
                        const uint2 x = __ldg(A.ent + ra.x + e);
                        const float2 rv = rho[x.x & kRay];
                        acc = fmaf(coef(x), __fadd_rn(rv.x, rv.y), acc);
                    }
                    if (heavy) {
#pragma unroll
                        for (int off = 16; off >= 8; off >>= 1) {
                            acc = __fadd_rn(acc, __shfl_xor_sync(kAllLanes, acc, off));
                            unlike += __shfl_xor_sync(kAllLanes, unlike, off);
                        }
                    }
#pragma unroll
                    for (int off = 4; off > 0; off >>= 1) {
                        acc = __fadd_rn(acc, __shfl_xor_sync(kAllLanes, acc, off));
                        unlike += __shfl_xor_sync(kAllLanes, unlike, off);
                    }
                    const float delta = xi ? -1.0f : 1.0f;
                    const float t = __fadd_rn(__uint_as_float(rb.x), acc);
                    const float prior = __fmul_rn(A.lambda, float(int(rb.w) - 2 * unlike));
                    const float dE = __fadd_rn(__fadd_rn(__fmul_rn(delta, t), __uint_as_float(rb.y)), prior);
                    const bool flip = live && (dE <= 0.0f || uphill_accept(u53, double(dE), T, inv_T));
                    if (flip) {
#pragma unroll
                        for (int u = 0; u < kHold; ++u)
                            rho[en[u].x & kRay] = two_sum_add(held[u], __fmul_rn(delta, __uint_as_float(en[u].y)));
                        for (int e = gl + G * kHold; e < rays; e += G) {
                            const uint2 x = __ldg(A.ent + ra.x + e);
                            float2& to = rho[x.x & kRay];
                            to = two_sum_add(to, __fmul_rn(delta, __uint_as_float(x.y)));
                        }
                        if (gl == 0) {
                            atomicXor(&xs[i >> 5], 1u << (i & 31));
                            ++my_accepts;
                            if (A.trace) atomicAdd(&s_trace, double(dE));
                        }
                    }
                } else {
                    const uint32_t tag = ra.y;
                    const int nsg = int(tag >> 16), base = 2 * int((tag >> 5) & 31u);
                    const int i = int(ra.z);
                    float2 held[kHold];
#pragma unroll
                    for (int u = 0; u < kHold; ++u) held[u] = rho[en[u].x & kRay];
                    const uint32_t xi = bit_of(i);
                    int unlike = 0;
#pragma unroll
                    for (int t = 0; t < kNbrLane; ++t)
                        if (nbr[t] >= 0) unlike += int(bit_of(nbr[t]) ^ xi);
                    const int gl = lane - base;
                    if (nsg && gl < 2)
                        for (int j = gl + 2 * kNbrLane; j < int(rb.w); j += 2) unlike += int(bit_of(__ldg(A.nbr + rb.z + j)) ^ xi);
                    float acc = 0.0f;
#pragma unroll
                    for (int u = 0; u < kHold; ++u) acc = fmaf(coef(en[u]), __fadd_rn(held[u].x, held[u].y), acc);
                    const float seg = __fadd_rn(acc, __shfl_xor_sync(kAllLanes, acc, 1));
                    unlike += __shfl_xor_sync(kAllLanes, unlike, 1);
                    unlike = __shfl_sync(kAllLanes, unlike, base);
                    // the bit's segment sums in order
                    const int most = int(__reduce_max_sync(kAllLanes, unsigned(nsg)));
                    float h = 0.0f;
                    for (int q0 = 0; q0 < min(most, kPairs); q0 += 4) {
                        float v[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = __shfl_sync(kAllLanes, seg, (base + 2 * (q0 + q)) & 31);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (q0 + q < min(nsg, kPairs)) h = __fadd_rn(h, v[q]);
                    }
                    // a bit of more segments has the warp to itself: further rounds
                    auto last_of = [&](int q) { return q == nsg - 1 ? int((tag >> 10) & 31u) : q < nsg ? kSegE : 0; };
                    for (int r = kPairs; r < most; r += kPairs) {
                        const int first = int(ra.x) + r * kSegE, l2 = last_of(r + pair);
                        float a2 = 0.0f;
                        for (int e = half; e < l2; e += 2) {
                            const uint2 en = __ldg(A.ent + first + e);
                            const float2 rv = rho[en.x & kRay];
                            a2 = fmaf(coef(en), __fadd_rn(rv.x, rv.y), a2);
                        }
                        const float s2 = __fadd_rn(a2, __shfl_xor_sync(kAllLanes, a2, 1));
                        for (int q = 0; q < min(most - r, kPairs); ++q) h = __fadd_rn(h, __shfl_sync(kAllLanes, s2, 2 * q));
                    }
                    const float delta = xi ? -1.0f : 1.0f;
                    const float t = __fadd_rn(__uint_as_float(rb.x), h);
                    const float prior = __fmul_rn(A.lambda, float(int(rb.w) - 2 * unlike));
                    const float dE = __fadd_rn(__fadd_rn(__fmul_rn(delta, t), __uint_as_float(rb.y)), prior);
                    const bool flip = nsg && (dE <= 0.0f || uphill_accept(u53, double(dE), T, inv_T));
                    if (flip) {
#pragma unroll
                        for (int u = 0; u < kHold; ++u)   // rho += delta a'
                            rho[en[u].x & kRay] = two_sum_add(held[u], __fmul_rn(delta, __uint_as_float(en[u].y)));
                        for (int r = kPairs; r < nsg; r += kPairs) {
                            const int first = int(ra.x) + r * kSegE, l2 = last_of(r + pair);
                            for (int e = half; e < l2; e += 2) {
                                const uint2 en = __ldg(A.ent + first + e);
                                float2& to = rho[en.x & kRay];
                                to = two_sum_add(to, __fmul_rn(delta, __uint_as_float(en.y)));
                            }
                        }
                        if (gl == 0) {
                            atomicXor(&xs[i >> 5], 1u << (i & 31));
                            ++my_accepts;
                            if (A.trace) atomicAdd(&s_trace, double(dE));
                        }
                    }
                }
                it0 += kLocalWarps;
                settle();
                if (s0 < A.sweeps) issue();
            } while (s0 == sweep && c0 == c);
            const bool last = c == nc - 1;
            if (last && (sweep + 1 == A.sweeps || full_stop(sweep + 1))) {
                ready = false;   // the whole CTA stops before the next class
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
    if (A.trace && tid == 0) A.trace[size_t(branch) * A.sweeps + A.sweeps - 1] = s_trace;
    for (int i = tid; i < n; i += kLocalThreads) A.x_out[size_t(branch) * size_t(n) + size_t(A.order[i])] = uint8_t(bit_of(i));
    if (my_accepts) atomicAdd(&s_accepts, my_accepts);
    __syncthreads();
    if (tid == 0 && s_accepts) atomicAdd(&A.accepts[0], s_accepts);
}

size_t local_smem(int n, int n_rays, int n_colours) {
    return (size_t(n_rays) + 1) * 8 + size_t((n + 31) / 32) * 4 + (size_t(n_colours) + 1) * 4;
}

}  // namespace

bool resid_local_fit(int n, int n_rays, int n_colours) { return n_rays >= 1 && local_smem(n, n_rays, n_colours) <= kLocalSmem; }

static void group_plan(ResidualPlan& P) {
    P.l_rec.clear();
    P.l_ptr.assign(1, 0);
    int items = 0;
    P.l_rec.reserve(size_t(P.n) * 9);
    auto put = [&](int k, int at, bool heavy) {
        uint32_t* r = &P.l_rec[(size_t(items - 1) * kGroupRecs + size_t(at)) * 8];
        const int row = P.h_row[size_t(k)];
        r[0] = uint32_t(row);
        r[1] = uint32_t(P.h_row[size_t(k) + 1] - row) | kLiveTag | (heavy ? kHeavyTag : 0u);
        r[2] = uint32_t(k);
        r[3] = uint32_t(P.col.order[size_t(k)]);
        std::memcpy(r + 4, &P.h_lin[size_t(k)], 4);
        std::memcpy(r + 5, &P.h_q[size_t(k)], 4);
        r[6] = uint32_t(P.h_nbr_ptr[size_t(k)]);
        r[7] = uint32_t(P.h_nbr_ptr[size_t(k) + 1] - P.h_nbr_ptr[size_t(k)]);
    };
    auto open_item = [&]() {
        ++items;
        P.l_rec.resize(size_t(items) * kGroupRecs * 8, 0u);
    };
    P.l_tail = P.l_long = 0.0;
    for (int c = 0; c < P.col.n_colours(); ++c) {
        int at = kGroupRecs, most = 0;
        for (int k = P.col.class_ptr[size_t(c)]; k < P.col.class_ptr[size_t(c) + 1]; ++k)
            if (P.h_row[size_t(k) + 1] - P.h_row[size_t(k)] > kHeavyRays) {
                open_item();
                for (int q = 0; q < kGroupRecs; ++q) put(k, q, true);
            }
        for (int k = P.col.class_ptr[size_t(c)]; k < P.col.class_ptr[size_t(c) + 1]; ++k) {
            if (P.h_row[size_t(k) + 1] - P.h_row[size_t(k)] > kHeavyRays) continue;
            if (at == kGroupRecs) {
                open_item();
                at = 0;
            }
            put(k, at++, false);
        }
        for (int k = P.col.class_ptr[size_t(c)]; k < P.col.class_ptr[size_t(c) + 1]; ++k)
            most = std::max(most, P.h_row[size_t(k) + 1] - P.h_row[size_t(k)]);
        P.l_tail += std::max(0, most - 32 * kHold);
        P.l_long += std::max(0, most - 1000);
        P.l_ptr.push_back(items);
    }
}

void resid_local_plan(ResidualPlan& P) {
    if (P.variant == QB_RESID_CLUSTER) return group_plan(P);
    P.l_rec.clear();
    P.l_ptr.assign(1, 0);
    const int nc = P.col.n_colours();
    auto segs = [&](int k) { return std::max(1, (P.h_row[size_t(k) + 1] - P.h_row[size_t(k)] + kSegE - 1) / kSegE); };
    int items = 0;
    P.l_rec.reserve((size_t(P.nnz) / kSegE + size_t(P.n)) * 8);
    auto open_item = [&]() {
        ++items;
        P.l_rec.resize(size_t(items) * kPairs * 8, 0u);
    };
    // bit k's pairs from pair `at` of the last item on
    auto put = [&](int k, int at) {
        const int row = P.h_row[size_t(k)], rays = P.h_row[size_t(k) + 1] - row, ns = segs(k);
        const int last = rays - (ns - 1) * kSegE;
        for (int j = 0; j < std::min(ns, kPairs); ++j) {
            uint32_t* r = &P.l_rec[(size_t(items - 1) * kPairs + size_t(at + j)) * 8];
            r[0] = uint32_t(row + j * kSegE);
            r[1] = rec_tag(j == ns - 1 ? last : kSegE, at, last, ns);
            r[2] = uint32_t(k);
            r[3] = uint32_t(P.col.order[size_t(k)]);
            std::copy_n(&P.h_meta[size_t(k) * 8 + 4], 2, r + 4);   // lin, q
            r[6] = uint32_t(P.h_nbr_ptr[size_t(k)]);
            r[7] = uint32_t(P.h_nbr_ptr[size_t(k) + 1] - P.h_nbr_ptr[size_t(k)]);
        }
    };
    std::vector<std::vector<int>> by(kPairs + 1);
    for (int c = 0; c < nc; ++c) {
        for (auto& v : by) v.clear();
        for (int k = P.col.class_ptr[size_t(c)]; k < P.col.class_ptr[size_t(c) + 1]; ++k) {
            const int ns = segs(k);
            if (ns > kPairs) {   // a warp item of its own
                open_item();
                put(k, 0);
            } else {
                by[size_t(ns)].push_back(k);
            }
        }
        // fill items with the largest bit that still fits
        for (;;) {
            int left = kPairs;
            while (left > 0) {
                int s = left;
                while (s > 0 && by[size_t(s)].empty()) --s;
                if (s == 0) break;
                if (left == kPairs) open_item();
                put(by[size_t(s)].back(), kPairs - left);
                by[size_t(s)].pop_back();
                left -= s;
            }
            if (left == kPairs) break;
        }
        P.l_ptr.push_back(items);
    }
}

// Microseconds per sweep, fitted to B200 times at 16 to 90,000 bits: a class
// step of the local sweep costs 1.05 or, once its items outnumber the warps,
// 0.1 per item; the lockstep sweep 3.9 per class at 16 branches and 13 % more
// per further 16 (90,000 bits: 16 branches 1.09 ms local, 0.88 lockstep; 64
// branches 1.09 and 1.22; 40,000 bits, 64 branches 0.54 and 0.83). Against the
// cluster sweep, in its order: a warp goes over a bit's rays beyond 256 and its
// neighbours beyond eight one load behind the other (100 bits of 1,000 rays, 16
// branches x 45 sweeps 28.0 ms local, 12.9 cluster; 1,000 bits of 48 neighbours,
// 149 branches 6.5 and 5.0), and a cluster CTA shares its SM with another.
bool resid_local_route(const ResidualPlan& p, int R) {
    if (!p.local || std::getenv("QB_PHASE_TIMES") || std::getenv("QB_TEST_BARRIER_STALL")) return false;
    const char* k = std::getenv("QB_RESID_KERNEL");
    if (k && (std::strcmp(k, "lockstep") == 0 || std::strcmp(k, "cluster") == 0)) return false;
    if (k && std::strcmp(k, "local") == 0) return true;
    // a forced cluster size asks for the cluster sweep
    const char* cl = std::getenv("QB_RESID_CLUSTER");
    if (p.variant == QB_RESID_CLUSTER && cl && *cl) return false;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const double classes = p.col.n_colours(), items = p.l_ptr.empty() ? 0.0 : p.l_ptr.back();
    const double local = std::max(1.05 * classes, 0.1 * items) * ((R + sms - 1) / sms);
    if (p.variant == QB_RESID_CLUSTER) {
        const double nbrs = 0.2 * std::max(0.0, double(p.n_nbr) / p.n / 8.0 - 1.0);
        const double one = std::max((1.05 + nbrs) * classes + 0.0069 * p.l_tail, 0.1 * items) * ((R + sms - 1) / sms);
        const double load = p.CL == 1 ? std::ceil(R / (2.0 * sms)) : std::max(1.0, R * p.CL / 100.0);
        return one < (3.3 * classes + 0.0035 * p.l_long) * load;
    }
    double lock = 0.0;
    for (int left = R; left > 0; left -= resid_lockstep_max_branches()) {
        const int groups = (std::min(left, resid_lockstep_max_branches()) + 15) / 16;
        lock += 3.9 * classes * (1.0 + 0.13 * (groups - 1));
    }
    return local < lock;
}

qb_status launch_resid_local(const ResidualPlan& p, const SolveBuffers& b, int R, int sweeps, int refresh, uint64_t seed0,
                             cudaStream_t st) {
    ResidLocalArgs A{};
    A.n = p.n;
    A.n_rays = p.n_rays;
    A.n_colours = p.col.n_colours();
    A.sweeps = sweeps;
    A.refresh = refresh;
    A.lambda = float(p.lambda);
    A.seed0 = seed0;
    A.rec = p.d_lrec.as<uint4>();
    A.item_ptr = p.d_lptr.as<int32_t>();
    A.ent = p.d_ent.as<uint2>();
    A.nbr = p.d_nbr_new.as<int32_t>();
    A.order = p.d_order.as<int32_t>();
    A.d = p.d_d.as<double>();
    A.w64 = p.d_w64.as<double>();
    A.rrow = p.d_rrow.as<int32_t>();
    A.rbit = p.d_rbit_new.as<int32_t>();
    A.ra = p.d_ra.as<float>();
    A.temp = b.temp;
    A.x_out = b.x;
    A.drift = b.drift;
    A.accepts = b.accepts;
    A.trace = b.trace;
    auto kern = p.variant == QB_RESID_CLUSTER ? resid_local_kernel<true> : resid_local_kernel<false>;
    QB_CUDA(allow_max_smem(kern));
    kern<<<unsigned(R), kLocalThreads, local_smem(p.n, p.n_rays, A.n_colours), st>>>(A);
    QB_CUDA(cudaGetLastError());
    count_sweep(p.variant == QB_RESID_CLUSTER ? Sweep::kResidLocalCluster : Sweep::kResidLocal);
    return QB_OK;
}

}  // namespace qb
