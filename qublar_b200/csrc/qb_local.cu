// Residual sweep with a CTA per branch: the branch's residual pairs and bits
// live in the CTA's shared memory (up to about 27,000 rays).
//
// The lockstep sweep (qb_kernels.cu) keeps all branches in global memory and
// closes every colour class with a grid barrier: about 4 us a class step
// whatever the class holds. Branches do not interact, so a branch that fits one
// SM needs no grid at all: a class step is gathers from shared memory and one
// CTA barrier.
//
// A warp item is 16 lane pairs, a pair per 16-entry segment of a bit (the even
// and the odd entries' fmaf chains, as in the lockstep sweep), a bit's pairs
// side by side: its segment sums are added in order through shuffles, every
// lane of the bit takes the decision, and each lane updates the residuals it
// holds -- no block barrier inside a class. A bit of more than 16 segments
// takes a warp to itself and goes over its segments in rounds. A warp's next
// item (record, entries, neighbour list, draw) is loaded while the current one
// runs; none of it depends on the state.
//
// Bound: the class step's chain (about 0.4 us) on small problems, the random
// 8-byte gathers from shared memory (about 5 lanes a cycle and SM, measured) on
// large ones.
//
// The arithmetic, the draws and hence the branches are the lockstep sweep's.
#include <cuda_runtime.h>

#include <algorithm>
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
constexpr int kLocalThreads = 512;
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
struct Rec {
    uint4 a, b;
};
__host__ __device__ inline uint32_t rec_tag(int len, int pair, int last, int segs) {
    return uint32_t(len) | uint32_t(pair) << 5 | uint32_t(last) << 10 | uint32_t(segs) << 16;
}

__global__ void __launch_bounds__(kLocalThreads, 1) resid_local_kernel(ResidLocalArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double s_trace;
    __shared__ unsigned long long s_accepts;
    const int nr = A.n_rays, n = A.n, nc = A.n_colours, words = (n + 31) / 32;
    float2* rho = reinterpret_cast<float2*>(smem);
    uint32_t* xs = reinterpret_cast<uint32_t*>(rho + nr);
    int32_t* ip = reinterpret_cast<int32_t*>(xs + words);
    const int tid = int(threadIdx.x), lane = tid & 31;
    const int warp = __shfl_sync(kAllLanes, tid >> 5, 0);
    const int pair = lane >> 1, half = lane & 1;
    const int branch = int(blockIdx.x);
    const uint64_t seed = A.seed0 + uint64_t(branch);
    for (int b = tid; b < nr; b += kLocalThreads) rho[b] = split_pair(-__dmul_rn(sqrt(fabs(A.w64[b])), A.d[b]));
    for (int k = tid; k < words; k += kLocalThreads) xs[k] = 0u;
    for (int c = tid; c <= nc; c += kLocalThreads) ip[c] = __ldg(A.item_ptr + c);
    if (tid == 0) {
        s_trace = 0.0;
        s_accepts = 0;
    }
    __syncthreads();

    auto bit_of = [&](int i) { return (xs[i >> 5] >> (i & 31)) & 1u; };
    auto rec_of = [&](int it) {
        const uint4* r = A.rec + (size_t(it) * kPairs + size_t(pair)) * 2;
        return Rec{__ldg(r), __ldg(r + 1)};
    };
    // the warp's items in visiting order: the next one of this class, else the
    // first of the next class that has one for it
    auto advance = [&](int& c, int& it, int& sweep) {
        it += kLocalWarps;
        if (it < ip[c + 1]) return;
        for (int k = 0; k < nc; ++k) {
            if (++c == nc) {
                c = 0;
                ++sweep;
            }
            it = ip[c] + warp;
            if (it < ip[c + 1]) return;
        }
        sweep = A.sweeps;   // no item at all
    };
    // what an item loads ahead besides its record
    uint2 ent[kHold];
    int nb[kNbrLane];
    uint64_t u53 = 0;
    auto fetch = [&](const Rec& r, int sweep) {
        const int len = int(r.a.y & 31u);
#pragma unroll
        for (int u = 0; u < kHold; ++u) {
            ent[u] = make_uint2(0u, 0u);
            if (half + 2 * u < len) ent[u] = __ldg(A.ent + r.a.x + half + 2 * u);
        }
        // lanes 0 and 1 of the bit share its neighbours
        const int gl = lane - 2 * int((r.a.y >> 5) & 31u);
#pragma unroll
        for (int t = 0; t < kNbrLane; ++t)
            nb[t] = (r.a.y >> 16) && gl < 2 && gl + 2 * t < int(r.b.w) ? __ldg(A.nbr + r.b.z + gl + 2 * t) : -1;
        u53 = draw_u53(seed, r.a.w, uint32_t(sweep), 0u);
    };
    auto coef = [](const uint2& e) { return (e.x >> 31) ? -__uint_as_float(e.y) : __uint_as_float(e.y); };

    // cur: the item in hand (its loads done or in flight); nx: the record after it
    int pc = 0, pit = ip[0] + warp - kLocalWarps, psw = 0;
    advance(pc, pit, psw);
    Rec cur{}, nx{};
    int c_at = pc, s_at = psw;
    if (psw < A.sweeps) {
        cur = rec_of(pit);
        fetch(cur, psw);
        advance(pc, pit, psw);
        if (psw < A.sweeps) nx = rec_of(pit);
    }
    unsigned long long my_accepts = 0;
    for (int sweep = 0; sweep < A.sweeps; ++sweep) {
        if (A.refresh > 0 && sweep > 0 && sweep % A.refresh == 0) {
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
            __syncthreads();
        }
        const double T = A.temp[sweep];
        const float inv_T = float(1.0 / T);
        for (int c = 0; c < nc; ++c) {
            while (s_at == sweep && c_at == c) {   // the warp's items of this class
                const uint32_t tag = cur.a.y;
                const int nsg = int(tag >> 16), base = 2 * int((tag >> 5) & 31u), len = int(tag & 31u);
                const int i = int(cur.a.z);
                // the residuals of the lane's entries
                float2 held[kHold];
#pragma unroll
                for (int u = 0; u < kHold; ++u) held[u] = rho[ent[u].x & kRay];   // entry 0 where there is none
                const uint32_t xi = nsg ? bit_of(i) : 0u;
                int unlike = 0;
#pragma unroll
                for (int t = 0; t < kNbrLane; ++t)
                    if (nb[t] >= 0) unlike += int(bit_of(nb[t]) ^ xi);
                const int gl = lane - base;
                if (nsg && gl < 2)
                    for (int j = gl + 2 * kNbrLane; j < int(cur.b.w); j += 2) unlike += int(bit_of(__ldg(A.nbr + cur.b.z + j)) ^ xi);
                float acc = 0.0f;
#pragma unroll
                for (int u = 0; u < kHold; ++u)
                    if (half + 2 * u < len) acc = fmaf(coef(ent[u]), __fadd_rn(held[u].x, held[u].y), acc);
                const float seg = __fadd_rn(acc, __shfl_xor_sync(kAllLanes, acc, 1));
                unlike += __shfl_xor_sync(kAllLanes, unlike, 1);
                unlike = __shfl_sync(kAllLanes, unlike, base);
                // the bit's segment sums in order
                const int most = int(__reduce_max_sync(kAllLanes, unsigned(nsg)));
                float h = 0.0f;
                for (int q = 0; q < min(most, kPairs); ++q) {
                    const float v = __shfl_sync(kAllLanes, seg, (base + 2 * q) & 31);
                    if (q < nsg) h = __fadd_rn(h, v);
                }
                // a bit of more segments has the warp to itself: further rounds
                auto last_of = [&](int q) { return q == nsg - 1 ? int((tag >> 10) & 31u) : q < nsg ? kSegE : 0; };
                for (int r = kPairs; r < most; r += kPairs) {
                    const int first = int(cur.a.x) + r * kSegE, l2 = last_of(r + pair);
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
                const float t = __fadd_rn(__uint_as_float(cur.b.x), h);
                const float prior = __fmul_rn(A.lambda, float(int(cur.b.w) - 2 * unlike));
                const float dE = __fadd_rn(__fadd_rn(__fmul_rn(delta, t), __uint_as_float(cur.b.y)), prior);
                const bool flip = nsg && (dE <= 0.0f || uphill_accept(u53, double(dE), T, inv_T));
                if (flip) {
#pragma unroll
                    for (int u = 0; u < kHold; ++u)
                        if (half + 2 * u < len)
                            rho[ent[u].x & kRay] = two_sum_add(held[u], __fmul_rn(delta, __uint_as_float(ent[u].y)));
                    for (int r = kPairs; r < nsg; r += kPairs) {
                        const int first = int(cur.a.x) + r * kSegE, l2 = last_of(r + pair);
                        for (int e = half; e < l2; e += 2) {
                            const uint2 en = __ldg(A.ent + first + e);
                            float2& at = rho[en.x & kRay];
                            at = two_sum_add(at, __fmul_rn(delta, __uint_as_float(en.y)));
                        }
                    }
                    if (gl == 0) {
                        atomicXor(&xs[i >> 5], 1u << (i & 31));
                        ++my_accepts;
                        if (A.trace) atomicAdd(&s_trace, double(dE));
                    }
                }
                // on to the next item: its record is here, its loads start
                cur = nx;
                c_at = pc;
                s_at = psw;
                if (psw < A.sweeps) {
                    fetch(cur, psw);
                    advance(pc, pit, psw);
                    if (psw < A.sweeps) nx = rec_of(pit);
                }
            }
            __syncthreads();
        }
        if (A.trace) {
            if (tid == 0) {
                A.trace[size_t(branch) * A.sweeps + sweep] = s_trace;
                s_trace = 0.0;
            }
            __syncthreads();
        }
    }
    for (int i = tid; i < n; i += kLocalThreads) A.x_out[size_t(branch) * size_t(n) + size_t(A.order[i])] = uint8_t(bit_of(i));
    if (my_accepts) atomicAdd(&s_accepts, my_accepts);
    __syncthreads();
    if (tid == 0 && s_accepts) atomicAdd(&A.accepts[0], s_accepts);
}

size_t local_smem(int n, int n_rays, int n_colours) {
    return size_t(n_rays) * 8 + size_t((n + 31) / 32) * 4 + (size_t(n_colours) + 1) * 4;
}

}  // namespace

bool resid_local_fit(int n, int n_rays, int n_colours) { return n_rays >= 1 && local_smem(n, n_rays, n_colours) <= kLocalSmem; }

void resid_local_plan(ResidualPlan& P) {
    P.l_rec.clear();
    P.l_ptr.assign(1, 0);
    const int nc = P.col.n_colours();
    auto segs = [&](int k) { return std::max(1, (P.h_row[size_t(k) + 1] - P.h_row[size_t(k)] + kSegE - 1) / kSegE); };
    int items = 0;
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

bool resid_local_route(const ResidualPlan& p) {
    if (!p.local) return false;
    const char* k = std::getenv("QB_RESID_KERNEL");
    return !(k && std::strcmp(k, "lockstep") == 0) && !std::getenv("QB_PHASE_TIMES") &&
           !std::getenv("QB_TEST_BARRIER_STALL");
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
    QB_CUDA(allow_max_smem(resid_local_kernel));
    resid_local_kernel<<<unsigned(R), kLocalThreads, local_smem(p.n, p.n_rays, A.n_colours), st>>>(A);
    QB_CUDA(cudaGetLastError());
    return QB_OK;
}

}  // namespace qb
