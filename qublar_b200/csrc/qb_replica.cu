// Integer Ising sweep of few replicas, or of a dense graph: a CTA anneals one
// replica with the random part of every decision taken off the sweep's chain.
//
// With no more replicas than SMs the time is the chain of colour classes
// (ER(800, 0.06): 17 classes x 1000 sweeps), not the work. So
//   * a draw u accepts every dE below -T ln u: its whole effect is one integer,
//     the largest dE it accepts (draw_limit_int, exact). Producer warps, or
//     helper CTAs of the replica's cluster that do nothing else, compute the
//     limits a few sweeps ahead into the replica's shared memory;
//   * a class step is dealt to few consumer warps: a lane per bit decides by
//     comparing two integers, and the accepted flips' rows are added to the
//     neighbours' fields by whole warps (few flips, long rows) or lane by lane;
//   * a bit's row, limit and spin do not change before its visit: they are
//     loaded before the barrier that opens its class, as is the CSR (in shared
//     memory where it fits).
//
// Bound: the dependent instructions of a class step in one warp (ncu, ER(800,
// 0.06), 16 replicas: 29 % issue on the SMs in use, barrier and fixed latencies;
// about 0.5 us against 0.74 of ising_anneal_kernel). Kernel time on
// a B200, before and after: ER(800, 0.06), 16 replicas x 1000 sweeps 12.4 and
// 8.5 ms; 3,001 bits of degree 8 with 32-bit couplings, 50 x 400: 2.4 and 1.8;
// complete graph of 16 spins, 32 x 100 (ising_dense_kernel below): 0.78 and
// 0.07. A form without fields, 16 lanes adding a bit's neighbours behind the
// barrier, was no faster (8.8 ms): its extra warps cost the issue slots that
// the atomics had.
//
// Fields, energies and decisions are those of ising_anneal_kernel
// (qb_kernels.cu), bit for bit.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>

#include "qb_device.cuh"
#include "qb_internal.hpp"
#include "qb_kernels.hpp"
#include "qb_philox.cuh"
#include "qb_word.hpp"

namespace cg = cooperative_groups;

namespace qb {

namespace {

constexpr unsigned kAllLanes = 0xffffffffu;
constexpr int kReplicaWarps = 32;

struct ReplicaArgs {
    int n;
    int n_colours;
    int nnz;
    int sweeps;
    int bound;       // max_i sum_j |w_ij|
    int consumers;   // warps
    int log2c;       // consumers = 1 << log2c
    int producers;   // warps of the replica's own CTA that draw
    int cluster;     // 1 + helper CTAs
    int ahead;       // sweeps drawn at a time
    int coop;        // a warp per accepted flip (else a lane per flip)
    int wbytes;
    uint64_t seed0;
    const int32_t* class_ptr;
    const int32_t* row;
    const int32_t* adj;
    const void* w;
    const int32_t* f0;
    const int32_t* order;
    const double* temp;
    uint8_t* x_out;
    int32_t* f_out;
    long long* e_out;
    long long* trace;
};

// The uphill test of an integer dE = k (uphill_accept's outcome).
__device__ __forceinline__ bool accept_int(uint64_t u53, int k, double T) {
    return double(u53) * 0x1.0p-53 < exp(-double(k) / T);
}

// The largest k in [0, bound] that the draw accepts: the test holds for k <
// X = -T ln u and fails beyond. In fp32, u = fp32(u53 2^-53) is within a
// relative 2^-23, so ln u within 2^-22.9 and the rounding of logf (1 ulp), the
// product and T add 2^-21 X: where X's distance from an integer exceeds T
// 2^-21 + X 2^-20, floor(X) is proven; otherwise the fp64 test of the nearest
// integer decides. X <= 36.8 T, so the margin stays below 0.17 for T <= 4096;
// above that X is taken in fp64 (error below (X + T) 2^-45, also the fp64
// test's own rounding) with the same structure; its last fallback, a margin above
// 1/4, is beyond the route's limit T <= 2^40 (X <= bound + 1 < 2^32: the margin
// stays below 2^-4). A zero draw searches.
__device__ __noinline__ int draw_limit_search(uint64_t u53, double T, int bound) {
    int lo = 0, hi = bound;   // accepted at lo
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (accept_int(u53, mid, T)) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int draw_limit_int(uint64_t u53, double T, float Tf, int bound) {
    if (u53 == 0) return draw_limit_search(u53, T, bound);
    if (Tf <= 4096.0f) {
        const float u = fmaf(float(uint32_t(u53) & 0x1FFFFFu), 0x1p-53f, float(uint32_t(u53 >> 21)) * 0x1p-32f);
        const float X = fmaxf(-logf(u) * Tf, 0.0f);
        const float err = fmaf(X, 0x1p-20f, Tf * 0x1p-21f);
        const float k = floorf(X), d = X - k;
        if (k > float(bound)) return bound;   // X exceeds the bound by more than err
        if (d > err && 1.0f - d > err) return min(int(k), bound);
        const int c = int(rintf(X));
        const int r = c == 0 || accept_int(u53, c, T) ? c : c - 1;
        return min(r, bound);
    }
    const double X = fmax(-log(double(u53) * 0x1.0p-53) * T, 0.0);
    if (X > double(bound) + 1.0) return bound;
    const double err = (X + T) * 0x1.0p-45, k = floor(X), d = X - k;
    if (d > err && 1.0 - d > err) return min(int(k), bound);
    if (err > 0.25) return draw_limit_search(u53, T, bound);
    const int c = int(rint(X));
    const int r = c == 0 || accept_int(u53, c, T) ? c : c - 1;
    return min(r, bound);
}

// Shared memory: limits[2][ahead][n], fields[n], row[n + 1], classes, weights
// and adjacency where they fit, spins.
template <typename WT, bool CSR>
__global__ void __launch_bounds__(32 * kReplicaWarps, 1) ising_replica_kernel(ReplicaArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long e_sum;
    const int n = A.n, nc = A.n_colours, S = A.ahead;
    int32_t* lim = reinterpret_cast<int32_t*>(smem);
    int32_t* f = lim + 2 * size_t(S) * size_t(n);
    int32_t* row = f + n;
    int32_t* cls = row + n + 1;
    WT* ws = reinterpret_cast<WT*>(cls + nc + 1);
    uint16_t* as = reinterpret_cast<uint16_t*>(smem + ((size_t(reinterpret_cast<unsigned char*>(ws + (CSR ? A.nnz : 0)) - smem) + 1) & ~size_t(1)));
    int8_t* s = reinterpret_cast<int8_t*>(as + (CSR ? A.nnz : 0));
    const int tid = int(threadIdx.x), threads = int(blockDim.x);
    const int lane = tid & 31, warp = __shfl_sync(kAllLanes, tid >> 5, 0);
    const int rep = int(blockIdx.x) / A.cluster, rank = int(blockIdx.x) - rep * A.cluster;
    const uint64_t key = ising_pair_key(A.seed0, uint32_t(rep));
    const int half = ising_pair_half(uint32_t(rep));
    uint32_t lim_base = uint32_t(__cvta_generic_to_shared(lim));
    if (A.cluster > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(lim_base) : "r"(lim_base), "r"(0));
    // the limits of sweeps s0 .. s0 + S - 1, blocks of 32 (sweep, bit) pairs
    // first, first + stride, ..., into the replica's CTA
    auto draw = [&](int s0, int first, int stride) {
        const int count = min(S, A.sweeps - s0) * n;
        const uint32_t base = lim_base + uint32_t((s0 / S) & 1) * uint32_t(S) * uint32_t(n) * 4u;
        for (int q = first * 32 + lane; q < count; q += stride * 32) {
            const int sl = S == 1 ? 0 : q / n, p = q - sl * n;
            const double T = A.temp[s0 + sl];
            const uint64_t u = draw_u53_half(key, uint32_t(__ldg(A.order + p)), uint32_t(s0 + sl), 0u, half);
            const int v = draw_limit_int(u, T, float(T), A.bound);
            if (A.cluster > 1) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(base + uint32_t(q) * 4u), "r"(v) : "memory");
            else lim[size_t((s0 / S) & 1) * size_t(S) * size_t(n) + q] = v;
        }
    };
    auto sync_all = [&]() {
        if (A.cluster > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    if (rank == 0) {
        for (int i = tid; i < n; i += threads) {
            f[i] = A.f0[i];
            s[i] = -1;
        }
        for (int i = tid; i <= n; i += threads) row[i] = A.row[i];
        for (int c = tid; c <= nc; c += threads) cls[c] = A.class_ptr[c];
        if (CSR)
            for (int k = tid; k < A.nnz; k += threads) {
                as[k] = uint16_t(A.adj[k]);
                ws[k] = static_cast<const WT*>(A.w)[k];
            }
        if (tid == 0) e_sum = 0;
    }
    const int own = threads >> 5, helpers = (A.cluster - 1) * own;
    // every warp of the cluster draws the first limits (once the whole cluster
    // is up: helpers write to the replica's CTA)
    sync_all();
    draw(0, rank * own + warp, own + helpers);
    sync_all();
    const WT* w = CSR ? ws : static_cast<const WT*>(A.w);
    auto adj_at = [&](int k) { return CSR ? int(as[k]) : __ldg(A.adj + k); };
    const bool consumer = rank == 0 && warp < A.consumers;
    const int32_t* limit = lim;
    // a visit's static part: its bit (or -1), spin, limit and row
    int i = -1, si = 0, li = 0, r0 = 0, r1 = 0;
    auto load = [&](int base, int c1) {   // the class's bits from base on, dealt in equal shares
        const int span = min(c1 - base, A.consumers * 32);
        const int per = (span + A.consumers - 1) >> A.log2c;
        i = lane < per && warp * per + lane < span ? base + warp * per + lane : -1;
        if (i >= 0) {
            si = s[i];
            li = limit[i];
            r0 = row[i];
            r1 = row[i + 1];
        }
    };
    long long E = 0;
    auto visit = [&]() {
        bool acc = false;
        if (i >= 0) {
            const int dE = -si * f[i];
            acc = dE <= li;
            if (acc) {
                s[i] = int8_t(-si);
                E += dE;
            }
        }
        // f_j -= 2 w_ij s_i, wrap-around uint32 (the final field fits int32, a
        // term may not)
        const uint32_t ms = si > 0 ? 0xFFFFFFFEu : 2u;
        if (A.coop) {
            unsigned m = __ballot_sync(kAllLanes, acc);
            while (m) {   // two flips, two stretches of 32 neighbours each at a time
                int k[2], k1[2];
                uint32_t mq[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int src = m ? __ffs(m) - 1 : 0;
                    const bool some = m != 0;
                    m &= m - 1u;
                    k[u] = __shfl_sync(kAllLanes, r0, src) + lane;
                    k1[u] = some ? __shfl_sync(kAllLanes, r1, src) : 0;
                    mq[u] = __shfl_sync(kAllLanes, ms, src);
                }
                do {
                    int j[4];
                    uint32_t d[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int q = k[u >> 1] + 32 * (u & 1);
                        j[u] = -1;
                        if (q < k1[u >> 1]) {
                            j[u] = adj_at(q);
                            d[u] = uint32_t(int32_t(w[q])) * mq[u >> 1];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j[u] >= 0) atomicAdd(reinterpret_cast<unsigned int*>(&f[j[u]]), d[u]);
                    k[0] += 64;
                    k[1] += 64;
                } while (__any_sync(kAllLanes, k[0] < k1[0] || k[1] < k1[1]));
            }
        } else if (acc) {
            int k = r0;
            for (; k + 4 <= r1; k += 4) {
                int j[4];
                uint32_t d[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    j[u] = adj_at(k + u);
                    d[u] = uint32_t(int32_t(w[k + u])) * ms;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) atomicAdd(reinterpret_cast<unsigned int*>(&f[j[u]]), d[u]);
            }
            for (; k < r1; ++k) atomicAdd(reinterpret_cast<unsigned int*>(&f[adj_at(k)]), uint32_t(int32_t(w[k])) * ms);
        }
    };
    for (int s0 = 0; s0 < A.sweeps; s0 += S) {
        if (!consumer) {
            if (s0 + S < A.sweeps)
                draw(s0 + S, rank == 0 ? warp - A.consumers : A.producers + (rank - 1) * own + warp, A.producers + helpers);
        } else {
            limit = lim + size_t((s0 / S) & 1) * size_t(S) * size_t(n);
            const int s1 = min(s0 + S, A.sweeps);
            const int stride = A.consumers * 32;
            load(0, cls[1]);
            for (int sweep = s0; sweep < s1; ++sweep) {
                int c0 = 0;
                for (int c = 0; c < nc; ++c) {
                    const int c1 = cls[c + 1];
                    visit();
                    for (int base = c0 + stride; base < c1; base += stride) {
                        load(base, c1);
                        visit();
                    }
                    // the next class's static part (of the next sweep behind the
                    // last class), then the barrier that opens it
                    if (c + 1 < nc) load(c1, cls[c + 2]);
                    else if (sweep + 1 < s1) {
                        limit += n;
                        load(0, cls[1]);   // one class: the lane that flipped a bit reloads it
                    }
                    c0 = c1;
                    asm volatile("bar.sync 1, %0;" ::"r"(A.consumers * 32) : "memory");
                }
                if (A.trace) {
                    long long Ew = E;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) Ew += __shfl_xor_sync(kAllLanes, Ew, off);
                    if (lane == 0 && Ew != 0)
                        atomicAdd(reinterpret_cast<unsigned long long*>(&A.trace[size_t(rep) * A.sweeps + sweep]),
                                  (unsigned long long)Ew);
                }
            }
        }
        sync_all();   // the next limits are in place, this block's are free
    }
    if (rank != 0) return;
    for (int p = tid; p < n; p += threads) {
        const size_t o = size_t(rep) * size_t(n) + size_t(A.order[p]);
        A.x_out[o] = s[p] > 0 ? 1u : 0u;
        A.f_out[o] = f[p];
    }
    if (consumer && E != 0) atomicAdd(&e_sum, (unsigned long long)E);
    __syncthreads();
    if (tid == 0) A.e_out[rep] = (long long)e_sum;
}

// Small graphs with many classes (dense ones): one warp holds the whole state
// in registers, lane l the fields of bits l, l + 32, ..., and visits the bits
// one by one in sweep order (the order inside a class does not matter), with
// the coupling matrix in shared memory. A visit is a multiply, a compare, a
// shuffle of the flip and a multiply-add: 50 to 95 ns by the bits a lane holds,
// against a class step through shared memory of 0.5 us and more. The other warps
// draw the limits kDenseAhead sweeps at a time.
constexpr int kDenseAhead = 8;
constexpr int kDenseMax = 224;   // bits: the matrix of 4-byte couplings fits shared memory

template <int K>
__global__ void __launch_bounds__(128) ising_dense_kernel(ReplicaArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = A.n;
    int32_t* W = reinterpret_cast<int32_t*>(smem);   // n x n
    int32_t* lim = W + size_t(n) * size_t(n);        // 2 x kDenseAhead x n
    const int tid = int(threadIdx.x), threads = int(blockDim.x), lane = tid & 31, warp = tid >> 5;
    const int rep = int(blockIdx.x);
    const uint64_t key = ising_pair_key(A.seed0, uint32_t(rep));
    const int half = ising_pair_half(uint32_t(rep));
    auto draw = [&](int s0, int t0, int stride) {
        int32_t* out = lim + size_t((s0 / kDenseAhead) & 1) * kDenseAhead * size_t(n);
        const int count = min(kDenseAhead, A.sweeps - s0) * n;
        for (int q = t0; q < count; q += stride) {
            const int sl = q / n, p = q - sl * n;
            const double T = A.temp[s0 + sl];
            const uint64_t u = draw_u53_half(key, uint32_t(__ldg(A.order + p)), uint32_t(s0 + sl), 0u, half);
            out[q] = draw_limit_int(u, T, float(T), A.bound);
        }
    };
    for (int k = tid; k < n * n; k += threads) W[k] = 0;
    draw(0, tid, threads);
    __syncthreads();
    for (int i = warp; i < n; i += threads >> 5)
        for (int k = __ldg(A.row + i) + lane; k < __ldg(A.row + i + 1); k += 32)
            W[i * n + __ldg(A.adj + k)] = A.wbytes == 1 ? int(static_cast<const int8_t*>(A.w)[k]) : static_cast<const int32_t*>(A.w)[k];
    __syncthreads();
    uint32_t f[K];
    int s[K];
    long long E = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        f[k] = 32 * k + lane < n ? uint32_t(A.f0[32 * k + lane]) : 0u;
        s[k] = -1;
    }
    for (int s0 = 0; s0 < A.sweeps; s0 += kDenseAhead) {
        if (warp > 0) {
            if (s0 + kDenseAhead < A.sweeps) draw(s0 + kDenseAhead, tid - 32, threads - 32);
        } else {
            const int32_t* in = lim + size_t((s0 / kDenseAhead) & 1) * kDenseAhead * size_t(n);
            const int s1 = min(s0 + kDenseAhead, A.sweeps);
            for (int sweep = s0; sweep < s1; ++sweep, in += n) {
                int limit[K];
#pragma unroll
                for (int k = 0; k < K; ++k) limit[k] = 32 * k + lane < n ? in[32 * k + lane] : -1;
#pragma unroll
                for (int b = 0; b < K; ++b) {
                    const int m = min(32, n - 32 * b);
                    const int32_t* w = W + size_t(32 * b) * size_t(n) + lane;
                    int wr[K];
#pragma unroll
                    for (int k = 0; k < K; ++k) wr[k] = m > 0 && 32 * k + lane < n ? w[32 * k] : 0;
                    for (int l = 0; l < m; ++l) {
                        const int dE = -s[b] * int(f[b]);
                        const bool a = dE <= limit[b];
                        const uint32_t ms = __shfl_sync(kAllLanes, a ? uint32_t(-2 * s[b]) : 0u, l);
                        w += n;
                        int wn[K];   // the next bit's row, off the chain
#pragma unroll
                        for (int k = 0; k < K; ++k) wn[k] = l + 1 < m && 32 * k + lane < n ? w[32 * k] : 0;
                        if (a && lane == l) {
                            s[b] = -s[b];
                            E += dE;
                        }
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            f[k] += uint32_t(wr[k]) * ms;   // f_j -= 2 w_ij s_i, wrap-around
                            wr[k] = wn[k];
                        }
                    }
                }
                if (A.trace) {
                    long long Ew = E;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) Ew += __shfl_xor_sync(kAllLanes, Ew, off);
                    if (lane == 0) A.trace[size_t(rep) * A.sweeps + sweep] = Ew;
                }
            }
        }
        __syncthreads();
    }
    if (warp > 0) return;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (32 * k + lane < n) {
            const size_t o = size_t(rep) * size_t(n) + size_t(A.order[32 * k + lane]);
            A.x_out[o] = s[k] > 0 ? 1u : 0u;
            A.f_out[o] = int32_t(f[k]);
        }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) E += __shfl_xor_sync(kAllLanes, E, off);
    if (lane == 0) A.e_out[rep] = E;
}

// A visit costs about an eighth of a class step: dense graphs, where most classes
// hold a few bits (above one replica per SM the route weighs its waves).
bool dense_fit(const IsingPlan& p) { return p.n <= kDenseMax && p.n <= 8 * p.col.n_colours(); }
size_t dense_smem(const IsingPlan& p) {
    return (size_t(p.n) * size_t(p.n) + 2 * size_t(kDenseAhead) * size_t(p.n)) * 4;
}

int replica_ahead(const IsingPlan& p) { return std::max(1, std::min(8, 4096 / p.n)); }
size_t replica_base_smem(const IsingPlan& p) {
    return size_t(p.n) * (8 * size_t(replica_ahead(p)) + 9) + size_t(p.col.n_colours() + 2) * 4 + 8;
}
size_t replica_csr_smem(const IsingPlan& p) { return size_t(p.nnz) * size_t(2 + p.weight_bytes); }
double replica_class(const IsingPlan& p) { return double(p.n) / std::max(1, p.col.n_colours()); }
// Consumer warps: a few bits of an average class each, so that the flips' rows
// are spread (ER(800, 0.06): 9.5 ms at 2 warps, 8.6 at 8, 9.1 at 16).
int replica_log2_consumers(const IsingPlan& p) {
    int l = 0;
    while (l < 4 && replica_class(p) > 6.0 * (1 << l)) ++l;
    return l;
}
// A warp per accepted flip while few of a warp's lanes can flip and rows are
// long (ER(800, 0.06): 8.6 ms against 20 with a lane per flip; 3,001 bits of
// degree 8: 2.4 ms against 1.8).
bool replica_coop(const IsingPlan& p) {
    const double per = std::ceil(replica_class(p) / (1 << replica_log2_consumers(p)));
    return 1.5 * per * ((p.max_deg + 31) / 32) < double(p.nnz) / p.n;
}
constexpr size_t kReplicaSmem = size_t(226) * 1024;
constexpr double kReplicaMaxT = 0x1.0p40;

// Clusters of `size` CTAs with an SM each that the device runs at once (a cluster
// stays within one GPC, so fewer than SMs / size), read once per device.
int cluster_room(int size) {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices][4];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices) return 0;
    std::atomic<int>& room = known[dev][size <= 2 ? 1 : size <= 4 ? 2 : 3];
    if (const int r = room.load(std::memory_order_relaxed)) return r;
    auto kern = ising_replica_kernel<int8_t, true>;
    if (allow_max_smem(kern) != cudaSuccess) return 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(size);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(size));
    cfg.blockDim = dim3(32 * kReplicaWarps);
    cfg.dynamicSmemBytes = kReplicaSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    room.store(n, std::memory_order_relaxed);
    return n;
}

// Cycles of a class step, and of a block of 32 draws in one warp (measured;
// only their ratio matters, for the number of helper CTAs).
constexpr double kStepCycles = 260.0, kDrawCycles = 1500.0;

}  // namespace

bool replica_csr_fit(const IsingPlan& p) { return replica_base_smem(p) + replica_csr_smem(p) <= kReplicaSmem; }

double dense_solve_us(const IsingPlan& p, int R, int sweeps) {
    // a visit takes 50, 65 or 95 ns by its registers; CTAs of an SM share it
    // from about nine on. 200 bits, 20 sweeps: 0.39 ms for 148 replicas, 1.91
    // for 600, 10.8 for 4,096 (CTA-per-replica sweep: 2.2, 2.3 and 7.2)
    const double visit = p.n <= 64 ? 0.050 : p.n <= 128 ? 0.065 : 0.095;
    const int fit = std::max(1, std::min(16, int(size_t(227) * 1024 / (dense_smem(p) + 1024))));
    const int waves = (R + word_sms() * fit - 1) / (word_sms() * fit);
    const double resident = std::min(double(fit), std::ceil(double(R) / word_sms()));
    return 8.0 + sweeps * (waves * p.n * visit * std::max(1.0, resident / 9.0));
}

// One wave of replicas (one CTA per SM) with the state in shared memory, or a
// dense graph. With the CSR in global memory only classes of at most a few
// hundred bits with a warp per flip and rows of up to 128 gain (2,000 bits of
// degree 120, 16 replicas x 50 sweeps: 1.82 ms against 2.15 for the
// CTA-per-replica sweep; ER(800, 0.5) 7.07 against 4.89; 10,000 bits of degree
// 40, classes of 600, 17.5 against 14.7). Where no SM is left for helper CTAs, wide classes
// of a small graph wait for the draws (1,600 bits in 2 classes, 148 replicas:
// 0.179 against 0.167; 4,225 in 4: 0.39 against 0.44). QB_ISING_THREADS asks for
// that sweep's CTA size, hence for that sweep.
bool replica_solve_fit(const IsingPlan& p, int R, double t_max) {
    if (t_max > kReplicaMaxT || std::getenv("QB_ISING_THREADS")) return false;
    if (dense_fit(p)) return true;
    if (R > word_sms() || replica_base_smem(p) > kReplicaSmem) return false;
    const bool helpers = 2 * R <= word_sms() && R <= cluster_room(2);
    if (!helpers && replica_class(p) > 300.0 && p.n < (p.weight_bytes == 1 ? 4200 : 6000)) return false;
    if (replica_csr_fit(p)) return true;
    return replica_class(p) <= 300.0 && p.nnz <= 128 * int64_t(p.n) && replica_coop(p);
}

qb_status launch_ising_replicas(const IsingPlan& p, const SolveBuffers& b, int R, int sweeps, uint64_t seed0,
                                cudaStream_t st) {
    ReplicaArgs A{};
    A.n = p.n;
    A.n_colours = p.col.n_colours();
    A.nnz = int(p.nnz);
    A.sweeps = sweeps;
    A.bound = int(p.B);
    A.seed0 = seed0;
    A.class_ptr = p.d_class_ptr.as<int32_t>();
    A.row = p.d_row.as<int32_t>();
    A.adj = p.d_adj.as<int32_t>();
    A.w = p.d_w.p;
    A.f0 = p.d_f0.as<int32_t>();
    A.order = p.d_order.as<int32_t>();
    A.temp = b.temp;
    A.x_out = b.x;
    A.f_out = b.f;
    A.e_out = b.e_i64;
    A.trace = reinterpret_cast<long long*>(b.trace);
    A.wbytes = p.weight_bytes;
    if (dense_fit(p)) {
        const size_t bytes = dense_smem(p);
        void (*kd)(ReplicaArgs) = p.n <= 32    ? ising_dense_kernel<1>
                                  : p.n <= 64  ? ising_dense_kernel<2>
                                  : p.n <= 128 ? ising_dense_kernel<4>
                                               : ising_dense_kernel<7>;
        QB_CUDA(allow_max_smem(kd));
        kd<<<unsigned(R), 128, bytes, st>>>(A);
        QB_CUDA(cudaGetLastError());
        count_sweep(Sweep::kIsingDense);
        return QB_OK;
    }
    A.log2c = replica_log2_consumers(p);
    A.consumers = 1 << A.log2c;
    A.coop = replica_coop(p) ? 1 : 0;
    const int blocks = (p.n + 31) / 32;
    A.ahead = replica_ahead(p);
    // helper CTAs where SMs are idle, as many as keep the drawing (about
    // kDrawCycles per 32 draws and warp) below the class steps; without them
    // the CTA's other warps draw. Only clusters that all run at once: 16 clusters
    // of 8 do not, and a second wave doubles the time (4,096 bits of a torus, 16
    // replicas x 40 sweeps: 0.36 ms, 0.19 for one replica)
    auto drawing = [&](int warps) { return kDrawCycles * std::ceil(double(A.ahead) * blocks / warps) / A.ahead; };
    const double steps = kStepCycles * A.n_colours;
    A.cluster = 1;
    if (drawing(kReplicaWarps - A.consumers) > steps)
        while (A.cluster < 8 && R * A.cluster * 2 <= word_sms() && R <= cluster_room(2 * A.cluster) &&
               (A.cluster == 1 || drawing(kReplicaWarps * (A.cluster - 1)) > steps))
            A.cluster *= 2;
    A.producers = A.cluster > 1 ? kReplicaWarps - A.consumers : std::min(kReplicaWarps - A.consumers, A.ahead * blocks);
    const bool csr = replica_csr_fit(p);
    const size_t smem = replica_base_smem(p) + (csr ? replica_csr_smem(p) : 0);
    void (*kern)(ReplicaArgs) = p.weight_bytes == 1 ? (csr ? ising_replica_kernel<int8_t, true> : ising_replica_kernel<int8_t, false>)
                                                    : (csr ? ising_replica_kernel<int32_t, true> : ising_replica_kernel<int32_t, false>);
    QB_CUDA(allow_max_smem(kern));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(R * A.cluster));
    cfg.blockDim = dim3(unsigned(32 * (A.consumers + A.producers)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(A.cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = A.cluster > 1 ? 1 : 0;
    QB_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    count_sweep(p.weight_bytes == 1 ? (csr ? Sweep::kIsingReplica8 : Sweep::kIsingReplica8Far)
                                    : (csr ? Sweep::kIsingReplica32 : Sweep::kIsingReplica32Far));
    return QB_OK;
}

}  // namespace qb
