// Integer Ising sweep for graphs of one coupling size (every |w_ij| = w0:
// unweighted and +-1 Max-Cut graphs, tori and d-regular +-1 graphs).
//
// A unit is G = 2 NP replicas of one instance; bit i's spins are one word of G
// bits in the CTA's shared memory and no field is kept: with v_j = x_j ^ x_i ^
// [w_ij < 0] a flip of i costs dE = w0 (2 c - deg) with c = #{j: v_j = 1}, so
// a visit counts its neighbours' words. A warp visits 32 / NP bits at once,
// lane (bit, pair p) serving replicas 2p and 2p + 1 (word bits p and p + NP),
// which share one Philox block. Sixteen neighbours of every bit are one
// register per lane: the NP lanes of a bit load 16 / NP words of G bits each,
// log2 NP butterfly rounds exchange neighbour and pair index between lanes and
// bit positions, and popcounts give the pair's counts.
//
// Bound: instruction issue, the half-rate integer pipe above all (ncu: 54 % of
// it, 59 % issue in units of 16 replicas, 51 and 56 in units of 32; 240 warp
// instructions per 64 proposals of degree 48, a quarter of them the Philox block,
// 25 per 16 neighbours). The field-carrying
// form (qb_batch.cu) spends an atomic per flipped neighbour and replica, and 5
// bytes of state per replica and bit against 1/4 here. Measured on a B200,
// kernel time: 4096 replicas x 300 sweeps of ER(800, 0.06) 16.6 ms with a CTA
// per replica, 6.4 ms here; 128 mixed tori and d-regular graphs of 200 to
// 20,000 bits, 32 replicas x 200 sweeps, 50 ms packed, 21.6 ms here (1.8e11
// proposals/s; 2.2e11 on 1,024 instances up to 5,000 bits).
//
// The CTA has 768 threads (one per SM: 80 registers each; at 64 the bodies
// spill) split into teams
// (named barriers) that run one unit each: large units take a whole CTA, small
// ones a quarter or an eighth, so that a unit's classes fill its warps.
//
// The decisions are those of the other integer sweeps: colour classes in
// order, accept if dE <= 0, else if u53 < ceil(exp(-dE / T) 2^53), u53 the
// draw half of (pair key, original bit, sweep).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "qb_batch.hpp"
#include "qb_device.cuh"
#include "qb_philox.cuh"
#include "qb_word.hpp"

namespace qb {

namespace {

constexpr unsigned kAll = 0xffffffffu;

static_assert(sizeof(WordItem) % 8 == 0, "WordItem is copied as 8-byte words");

template <int G>
struct WordOf;
template <> struct WordOf<32> { using T = uint32_t; };
template <> struct WordOf<16> { using T = uint16_t; };
template <> struct WordOf<8> { using T = uint8_t; };
template <> struct WordOf<4> { using T = uint8_t; };

// The bit positions of replicas 2p of the butterfly's result (see count_pair).
template <int NP>
__device__ __forceinline__ constexpr unsigned low_mask() {
    return NP == 16 ? 0x0000FFFFu : NP == 8 ? 0x00FF00FFu : NP == 4 ? 0x0F0F0F0Fu : 0x33333333u;
}

constexpr int kMaxTeams = 8;

struct Team {
    int id;        // named barrier
    int tid;       // thread in the team
    int threads;
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
    }
};

// u53 < t as a test on the draw's 64 bits with the low 11 cleared.
__device__ __forceinline__ unsigned long long draw_limit(int k, double T) {
    const double p = exp(-double(k) / T);
    const unsigned long long t = (unsigned long long)ceil(p * 0x1.0p53);
    return t >= (1ull << 53) ? ~0ull : t << 11;
}

// The butterfly that turns "sixteen neighbours' words" into "sixteen
// neighbours' bits per replica": register bit t G + pos of lane q is replica
// position pos of neighbour (q, t) of its bit; each round swaps one bit of the
// lane index with one of the position. Afterwards the bits of low_mask are the
// neighbours in replica 2p of lane p, the others those in replica 2p + 1.
template <int NP>
struct Butterfly {
    static constexpr int kRounds = NP == 16 ? 4 : NP == 8 ? 3 : NP == 4 ? 2 : 1;
    uint32_t keep[kRounds];
    int rot[kRounds];
    __device__ __forceinline__ explicit Butterfly(int q) {
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            const int j = NP >> (r + 1);
            const unsigned L = j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u : 0x55555555u;
            const bool up = (q & j) != 0;
            keep[r] = up ? ~L : L;
            rot[r] = up ? 32 - j : j;
            asm volatile("" : "+r"(keep[r]), "+r"(rot[r]));   // kept in registers: three instructions a round
        }
    }
    // K registers go through together, so that their shuffles overlap.
    template <int K>
    __device__ __forceinline__ void apply(uint32_t (&v)[K]) const {
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            uint32_t o[K];
#pragma unroll
            for (int u = 0; u < K; ++u) o[u] = __shfl_xor_sync(kAll, v[u], NP >> (r + 1));
#pragma unroll
            for (int u = 0; u < K; ++u)   // bits that wrap are masked off
                v[u] = (v[u] & keep[r]) | (__funnelshift_l(o[u], o[u], rot[r]) & ~keep[r]);
        }
    }
};

// Where a sweep's words live: the CTA's shared memory, or global memory that
// other CTAs write (read past the L1 cache).
template <typename WT>
struct SharedWords {
    const WT* p;
    __device__ __forceinline__ uint32_t operator[](uint32_t j) const { return uint32_t(p[j]); }
};
struct GlobalWords {
    const uint32_t* p;
    __device__ __forceinline__ uint32_t operator[](uint32_t j) const { return __ldcg(p + j); }
};

// A lane's share of one chunk of sixteen neighbours: 16 / NP consecutive
// entries, loaded at once. Rows are padded to sixteen with the bit itself,
// whose word cancels; a chunk past the row is the bit itself throughout.
template <int NP, typename AT>
struct Share {
    static constexpr int E = 16 / NP;                                             // entries
    static constexpr int W = E * int(sizeof(AT)) > 4 ? E * int(sizeof(AT)) / 4 : 1;   // registers
    uint32_t w[W];
    __device__ __forceinline__ void load(const AT* __restrict__ row, int u, int deg, uint32_t self) {
        const bool in = 16 * u < deg;
        if (W == 1) {
            w[0] = self;
            if (in)
                w[0] = E * sizeof(AT) == 2 ? uint32_t(__ldg(row + 16 * u)) : __ldg(reinterpret_cast<const uint32_t*>(row + 16 * u));
        } else {
#pragma unroll
            for (int t = 0; t < W; t += 2) {
                uint2 p = make_uint2(self, self);
                if (in) p = __ldg(reinterpret_cast<const uint2*>(row + 16 * u + t * 4 / int(sizeof(AT))));
                w[t] = p.x;
                w[W > 1 ? t + 1 : 0] = p.y;
            }
        }
    }
    // The neighbours' words against the bit's own (xr: repeated over the register), packed.
    template <typename XS>
    __device__ __forceinline__ uint32_t words(const XS& X, uint32_t xr) const {
        constexpr int G = 2 * NP;
        uint32_t v = 0;
#pragma unroll
        for (int t = 0; t < E; ++t) {
            const uint32_t e = sizeof(AT) == 4 || E == 1 ? w[t < W ? t : 0] : t & 1 ? w[t / 2] >> 16 : w[t / 2] & 0xFFFFu;
            v += X[e] << (t * G);
        }
        return v ^ xr;
    }
};

// Chunks of the next pass loaded ahead: three or four registers.
template <int NP, typename AT>
struct Ahead {
    static constexpr int K = Share<NP, AT>::W == 1 ? 4 : Share<NP, AT>::W == 2 ? 2 : 1;
    Share<NP, AT> s[K];
    // row: the lane's first entry; self: the bit, packed as entries are
    __device__ __forceinline__ void load(const AT* __restrict__ row, int deg, uint32_t self) {
#pragma unroll
        for (int u = 0; u < K; ++u) s[u].load(row, u, deg, self);
    }
};

// The bit's own index as a register of a share holds entries: two 16-bit ones,
// or a single entry (a 32-bit one, or the only one of NP = 16).
template <int NP, typename AT>
__device__ __forceinline__ uint32_t packed_self(int i) {
    return sizeof(AT) == 2 && NP < 16 ? uint32_t(i) * 0x00010001u : uint32_t(i);
}

// A word of G bits repeated over the register.
template <int G>
__device__ __forceinline__ uint32_t repeated(uint32_t x) {
    return G == 32 ? x : x * (G == 16 ? 0x00010001u : G == 8 ? 0x01010101u : 0x11111111u);
}

template <int NP>
__device__ __forceinline__ void add_counts(uint32_t v, int weight, int& ca, int& cb) {
    ca += weight * __popc(v & low_mask<NP>());
    cb += weight * __popc(v & ~low_mask<NP>());
}

// Counts of K chunks' packed words; three or four go through the butterfly as
// two or three registers, added bit by bit first (full adders).
template <int NP, int K>
__device__ __forceinline__ void count_chunks(const Butterfly<NP>& bf, const uint32_t (&v)[K], int& ca, int& cb) {
    if constexpr (K <= 2) {
        uint32_t t[K];
#pragma unroll
        for (int u = 0; u < K; ++u) t[u] = v[u];
        bf.apply(t);
#pragma unroll
        for (int u = 0; u < K; ++u) add_counts<NP>(t[u], 1, ca, cb);
    } else {
        const uint32_t s = v[0] ^ v[1] ^ v[2], m = (v[0] & v[1]) | (v[2] & (v[0] | v[1]));
        if constexpr (K == 3) {
            uint32_t t[2] = {s, m};
            bf.apply(t);
            add_counts<NP>(t[0], 1, ca, cb);
            add_counts<NP>(t[1], 2, ca, cb);
        } else {
            uint32_t t[3] = {s ^ v[3], m, s & v[3]};
            bf.apply(t);
            add_counts<NP>(t[0], 1, ca, cb);
            add_counts<NP>(t[1], 2, ca, cb);
            add_counts<NP>(t[2], 2, ca, cb);
        }
    }
}

template <int NP, int K, typename AT, typename XS>
__device__ __forceinline__ void count_ahead(const Butterfly<NP>& bf, const Ahead<NP, AT>& ah, const XS& X, uint32_t xr,
                                            int& ca, int& cb) {
    uint32_t v[K];
#pragma unroll
    for (int u = 0; u < K; ++u) v[u] = ah.s[u].words(X, xr);
    count_chunks<NP, K>(bf, v, ca, cb);
}

// For the warp's bits (lane = (bit, pair p)): the number of neighbours j of
// bit i with v_j = 1 in replicas 2p (ca) and 2p + 1 (cb). The first chunks'
// entries are in `ah`.
template <int NP, typename AT, typename XS>
__device__ __forceinline__ void count_pair(const Butterfly<NP>& bf, const XS& X, const AT* __restrict__ row, int deg,
                                           uint32_t self, uint32_t xi, const Ahead<NP, AT>& ah, int& ca, int& cb) {
    constexpr int K = Ahead<NP, AT>::K;
    const uint32_t xr = repeated<2 * NP>(xi);
    const int chunks = (__reduce_max_sync(kAll, deg) + 15) >> 4;
    ca = cb = 0;
    if (K == 1 || chunks <= 1) count_ahead<NP, 1, AT, XS>(bf, ah, X, xr, ca, cb);
    else if (K == 2 || chunks == 2) count_ahead<NP, (K > 1 ? 2 : 1), AT, XS>(bf, ah, X, xr, ca, cb);
    else if (chunks == 3) count_ahead<NP, (K > 2 ? 3 : 1), AT, XS>(bf, ah, X, xr, ca, cb);
    else count_ahead<NP, K, AT, XS>(bf, ah, X, xr, ca, cb);
    for (int u = K; u < chunks; u += 3) {   // longer rows: three chunks at a time
        Share<NP, AT> s[3];
#pragma unroll
        for (int t = 0; t < 3; ++t) s[t].load(row, u + t, deg, self);
        uint32_t v[3];
#pragma unroll
        for (int t = 0; t < 3; ++t) v[t] = s[t].words(X, xr);
        count_chunks<NP, 3>(bf, v, ca, cb);
    }
}

// Dynamic shared memory: the header, then one share per team.
struct WordHead {
    WordItem it[kMaxTeams];
    long long e[kMaxTeams][32];
    int next;
    int pad[3];
};
static_assert(sizeof(WordHead) % 16 == 0, "the shares follow the header");

extern __shared__ __align__(16) unsigned char word_smem[];

template <int NP, typename AT>
__device__ __forceinline__ void word_item(int team, int tid, int threads, uint32_t share_off) {
    constexpr int G = 2 * NP;
    constexpr int BW = 32 / NP;   // bits per warp pass
    constexpr uint32_t kG = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    using WT = typename WordOf<G>::T;
    WordHead* head = reinterpret_cast<WordHead*>(word_smem);
    const WordItem& it = head->it[team];
    long long* e_sh = head->e[team];
    const Team tm{1 + team, tid, threads};
    const int n = it.n, nc = it.n_colours, max_deg = it.max_deg;
    // limits of 2 c - deg = -max_deg .. max_deg: every move that does not raise
    // the energy passes
    unsigned long long* thr = reinterpret_cast<unsigned long long*>(word_smem + share_off) + max_deg;
    int32_t* cls = reinterpret_cast<int32_t*>(thr + max_deg + 1);
    WT* X = reinterpret_cast<WT*>(cls + nc + 1);   // n words, then their complements
    const int lane = int(threadIdx.x & 31u);
    const int q = lane & (NP - 1);
    const int sub = lane / NP;
    const int warp = __shfl_sync(kAll, tid >> 5, 0), warps = threads >> 5;
    const AT* __restrict__ adj = static_cast<const AT*>(it.adj);
    const uint4* __restrict__ recs = it.rec;
    const int flags = it.flags;
    if (flags & kItemInit) {
        for (int i = tid; i < n; i += threads) {
            X[i] = 0;
            X[n + i] = WT(kG);
        }
    } else {
        const WT* kept = static_cast<const WT*>(it.state);
        for (int i = tid; i < n; i += threads) {
            X[i] = kept[i];
            X[n + i] = WT(kept[i] ^ kG);
        }
    }
    for (int c = tid; c <= nc; c += threads) cls[c] = __ldg(it.class_ptr + c);
    for (int m = tid; m <= max_deg; m += threads) thr[-m] = ~0ull;
    tm.sync();
    const uint64_t key = it.seed0 + uint64_t(2 * q);
    // the record and the first chunks of the warp's next pass are loaded while
    // the current one runs (the structure does not depend on the state)
    auto bit_at = [&](int base, int c1) { return min(base + sub, c1 - 1); };
    auto row_of = [&](const uint4& r) { return adj + size_t(r.x) * 16 + q * Share<NP, AT>::E; };
    const Butterfly<NP> bf(q);
    uint4 rec = make_uint4(0u, 0u, 0u, 0u);
    Ahead<NP, AT> ah;
    int ready = -1;   // the base that rec and ah hold
    const int sweep1 = it.sweep1;
    for (int sweep = it.sweep0; sweep < sweep1; ++sweep) {
        const double T = it.temp[sweep];
        for (int m = tid + 1; m <= max_deg; m += threads) thr[m] = draw_limit(it.w0 * m, T);
        tm.sync();
        for (int c = 0; c < nc; ++c) {
            const int c1 = cls[c + 1];
            for (int base = cls[c] + warp * BW; base < c1; base += warps * BW) {
                const int i = bit_at(base, c1);
                const bool valid = base + sub < c1;
                if (ready != base) {   // nothing loaded ahead (the first pass, or a class without one)
                    rec = __ldg(recs + i);
                    ah.load(row_of(rec), int(rec.y), packed_self<NP, AT>(i));
                }
                // the next pass: in this class, else the next class's first
                int nb = base + warps * BW, n1 = c1;
                if (nb >= c1) {
                    const int cn = c + 1 < nc ? c + 1 : 0;
                    nb = cls[cn] + warp * BW;
                    n1 = cls[cn + 1];
                }
                const bool more = nb < n1;
                const int ni = more ? bit_at(nb, n1) : i;
                const uint4 rn = __ldg(recs + ni);
                const int deg = int(rec.y);
                const uint32_t xi = uint32_t(X[i]);
                int ca, cb;
                count_pair<NP, AT>(bf, SharedWords<WT>{X}, row_of(rec), deg, packed_self<NP, AT>(i), xi, ah, ca, cb);
                const uint32_t oi = rec.z;
                rec = rn;
                ah.load(row_of(rec), int(rec.y), packed_self<NP, AT>(ni));
                ready = more ? nb : -1;
                const unsigned long long ta = thr[2 * ca - deg], tb = thr[2 * cb - deg];
                const Philox4 d = philox4x32_10(oi, uint32_t(sweep), 0u, 0u, uint32_t(key), uint32_t(key >> 32));
                const unsigned long long za = (uint64_t(d.v[1]) << 32) | uint64_t(d.v[0] & ~2047u);
                const unsigned long long zb = (uint64_t(d.v[3]) << 32) | uint64_t(d.v[2] & ~2047u);
                const unsigned ba = __ballot_sync(kAll, valid && za < ta), bb = __ballot_sync(kAll, valid && zb < tb);
                if (q == 0 && valid) {
                    constexpr unsigned kP = (1u << NP) - 1u;
                    const unsigned flip = NP == 16 ? __byte_perm(ba, bb, sub ? 0x7632 : 0x5410)
                                          : NP == 8 ? __byte_perm(ba, bb, sub * 0x11 + 0x40)
                                                    : ((ba >> (sub * NP)) & kP) | (((bb >> (sub * NP)) & kP) << NP);
                    X[i] = WT((xi ^ flip) & kG);
                    X[n + i] = WT(~(xi ^ flip) & kG);
                }
            }
            tm.sync();
        }
    }
    if (flags & kItemKeep) {
        WT* kept = static_cast<WT*>(it.state);
        for (int i = tid; i < n; i += threads) kept[i] = X[i];
    }
    if (flags & kItemFinal) {
        // fields and energies from the final words: f_i = w0 (2 c - deg) for x_i
        // = 0 and its negative for x_i = 1, E = (sum_i s_i f_i + sum_i f0_i) / 4
        // (the sum of the accepted dE, exactly: all integers)
        if (tid < 32) e_sh[tid] = 0;
        tm.sync();
        long long Ea = 0, Eb = 0;
        const int ra = 2 * q, rb = 2 * q + 1, live = it.live, w0 = it.w0;
        uint8_t* x_out = it.x_out;
        int32_t* f_out = it.f_out;
        for (int base = warp * BW; base < n; base += warps * BW) {
            const bool valid = base + sub < n;
            const int i = bit_at(base, n);
            rec = __ldg(recs + i);
            ah.load(row_of(rec), int(rec.y), packed_self<NP, AT>(i));
            const int deg = int(rec.y);
            const uint32_t xi = uint32_t(X[i]);
            int ca, cb;
            count_pair<NP, AT>(bf, SharedWords<WT>{X}, row_of(rec), deg, packed_self<NP, AT>(i), xi, ah, ca, cb);
            if (valid) {
                const size_t o = size_t(rec.z);
                const int da = w0 * (2 * ca - deg), db = w0 * (2 * cb - deg);   // = -s_i f_i
                const int xa = int((xi >> q) & 1u), xb = int((xi >> (q + NP)) & 1u);
                Ea -= da;
                Eb -= db;
                if (ra < live) {
                    x_out[size_t(ra) * size_t(n) + o] = uint8_t(xa);
                    f_out[size_t(ra) * size_t(n) + o] = xa ? -da : da;
                }
                if (rb < live) {
                    x_out[size_t(rb) * size_t(n) + o] = uint8_t(xb);
                    f_out[size_t(rb) * size_t(n) + o] = xb ? -db : db;
                }
            }
        }
        atomicAdd(reinterpret_cast<unsigned long long*>(&e_sh[ra]), (unsigned long long)Ea);
        atomicAdd(reinterpret_cast<unsigned long long*>(&e_sh[rb]), (unsigned long long)Eb);
        tm.sync();
        if (tid < live) it.e_out[tid] = (e_sh[tid] + it.f0_sum) / 4;
    }
}

// The adjacency's width is the kernel's: with both widths' bodies in one
// kernel the register allocation spills.
template <typename AT>
__global__ void __launch_bounds__(kWordThreads, 1) ising_word_kernel(const WordItem* __restrict__ items,
                                                                     const WordBundle* __restrict__ bundles,
                                                                     int n_bundles, int* counter) {
    WordHead* head = reinterpret_cast<WordHead*>(word_smem);
    for (;;) {
        if (threadIdx.x == 0) head->next = atomicAdd(counter, 1);
        __syncthreads();
        const int k = head->next;
        if (k >= n_bundles) return;
        const WordBundle b = bundles[k];
        constexpr int kWords = int(sizeof(WordItem) / 8);
        for (int w = int(threadIdx.x); w < b.count * kWords; w += kWordThreads)
            reinterpret_cast<uint64_t*>(head->it)[w] = reinterpret_cast<const uint64_t*>(items + b.first)[w];
        __syncthreads();
        const int threads = kWordThreads / b.teams;
        const int t = int(threadIdx.x) / threads;
        if (t < b.count) {
            const uint32_t off = uint32_t(sizeof(WordHead)) + uint32_t(t) * uint32_t(b.share);
            const int tid = int(threadIdx.x) - t * threads;
            switch (head->it[t].log2np) {
                case 4: word_item<16, AT>(t, tid, threads, off); break;
                case 3: word_item<8, AT>(t, tid, threads, off); break;
                case 2: word_item<4, AT>(t, tid, threads, off); break;
                default: word_item<2, AT>(t, tid, threads, off); break;
            }
        }
        __syncthreads();
    }
}

// One problem on the whole device: words of 32 replicas in global memory, a
// cooperative grid whose warps visit a class's bits (two per pass) for every
// group of 32 replicas, a bounded grid barrier behind each class. For few
// replicas of a large graph, where a CTA per replica leaves most SMs idle.
// Bound: the class step's latency, a grid barrier (1.4 us) and the pass behind
// it (L2 gathers). 60,000 bits of degree 5, 32 replicas x 100 sweeps on a B200:
// 15.5 ms with a CTA per replica, 2.9 here.
struct GridArgs {
    const int32_t* class_ptr;
    const uint4* rec;
    const void* adj;
    const double* temp;
    uint32_t* X;          // groups x 2 n words: values, complements
    long long* e_out;     // R (zeroed)
    uint8_t* x_out;
    int32_t* f_out;
    unsigned* bar;
    int* err;
    uint64_t seed0;
    long long f0_sum;
    int n;
    int n_colours;
    int sweeps;
    int R;
    int groups;
    int w0;
    int max_deg;
};

constexpr int kGridThreads = 1024;

template <typename AT>
__global__ void __launch_bounds__(kGridThreads, 1) ising_grid_kernel(GridArgs A) {
    constexpr int NP = 16, BW = 2;
    __shared__ unsigned long long s_thr[2 * kWordMaxDegree + 1];
    __shared__ long long s_e[32];
    const int n = A.n, nc = A.n_colours, max_deg = A.max_deg;
    unsigned long long* thr = s_thr + max_deg;
    const int tid = int(threadIdx.x), lane = tid & 31, q = lane & (NP - 1), sub = lane / NP;
    const int gw = __shfl_sync(kAll, int(blockIdx.x) * (kGridThreads / 32) + (tid >> 5), 0);
    const int tw = int(gridDim.x) * (kGridThreads / 32);
    const AT* __restrict__ adj = static_cast<const AT*>(A.adj);
    const Butterfly<NP> bf(q);
    auto row_of = [&](const uint4& r) { return adj + size_t(r.x) * 16 + q; };
    for (size_t k = size_t(blockIdx.x) * kGridThreads + tid; k < size_t(A.groups) * 2 * size_t(n);
         k += size_t(gridDim.x) * kGridThreads)
        __stcg(A.X + k, (k / size_t(n)) & 1 ? kAll : 0u);
    for (int m = tid; m <= max_deg; m += kGridThreads) thr[-m] = ~0ull;
    unsigned round = 0;
    bool ok = grid_barrier(A.bar, A.err, ++round);
    Ahead<NP, AT> ah;
    for (int sweep = 0; ok && sweep < A.sweeps; ++sweep) {
        const double T = A.temp[sweep];
        for (int m = tid + 1; m <= max_deg; m += kGridThreads) thr[m] = draw_limit(A.w0 * m, T);
        __syncthreads();
        for (int c = 0; ok && c < nc; ++c) {
            const int c0 = __ldg(A.class_ptr + c), c1 = __ldg(A.class_ptr + c + 1);
            const int passes = (c1 - c0 + BW - 1) / BW;
            for (int p = gw; p < passes * A.groups; p += tw) {
                const int g = p / passes, base = c0 + (p - g * passes) * BW;
                const bool valid = base + sub < c1;
                const int i = valid ? base + sub : c1 - 1;
                const uint4 rec = __ldg(A.rec + i);
                const int deg = int(rec.y);
                const uint32_t self = packed_self<NP, AT>(i);
                ah.load(row_of(rec), deg, self);
                uint32_t* X = A.X + size_t(g) * 2 * size_t(n);
                const uint32_t xi = __ldcg(X + i);
                const uint64_t key = A.seed0 + uint64_t(32 * g) + uint64_t(2 * q);
                const Philox4 d = philox4x32_10(rec.z, uint32_t(sweep), 0u, 0u, uint32_t(key), uint32_t(key >> 32));
                int ca, cb;
                count_pair<NP, AT>(bf, GlobalWords{X}, row_of(rec), deg, self, xi, ah, ca, cb);
                const unsigned long long za = (uint64_t(d.v[1]) << 32) | uint64_t(d.v[0] & ~2047u);
                const unsigned long long zb = (uint64_t(d.v[3]) << 32) | uint64_t(d.v[2] & ~2047u);
                const unsigned ba = __ballot_sync(kAll, valid && za < thr[2 * ca - deg]);
                const unsigned bb = __ballot_sync(kAll, valid && zb < thr[2 * cb - deg]);
                if (q == 0 && valid) {
                    const uint32_t x = xi ^ __byte_perm(ba, bb, sub ? 0x7632 : 0x5410);
                    __stcg(X + i, x);
                    __stcg(X + n + i, ~x);
                }
            }
            ok = grid_barrier(A.bar, A.err, ++round);
        }
    }
    if (!ok) return;
    // fields and energies from the final words, as in word_item
    const int passes = (n + BW - 1) / BW;
    for (int g = 0; g < A.groups; ++g) {
        if (tid < 32) s_e[tid] = 0;
        __syncthreads();
        const int ra = 32 * g + 2 * q, rb = ra + 1;
        long long Ea = 0, Eb = 0;
        for (int p = gw; p < passes; p += tw) {
            const bool valid = p * BW + sub < n;
            const int i = valid ? p * BW + sub : n - 1;
            const uint4 rec = __ldg(A.rec + i);
            const int deg = int(rec.y);
            const uint32_t self = packed_self<NP, AT>(i);
            ah.load(row_of(rec), deg, self);
            const uint32_t* X = A.X + size_t(g) * 2 * size_t(n);
            const uint32_t xi = __ldcg(X + i);
            int ca, cb;
            count_pair<NP, AT>(bf, GlobalWords{X}, row_of(rec), deg, self, xi, ah, ca, cb);
            if (!valid) continue;
            const size_t o = size_t(rec.z);
            const int da = A.w0 * (2 * ca - deg), db = A.w0 * (2 * cb - deg);
            const int xa = int((xi >> q) & 1u), xb = int((xi >> (q + NP)) & 1u);
            Ea -= da;
            Eb -= db;
            if (ra < A.R) {
                A.x_out[size_t(ra) * size_t(n) + o] = uint8_t(xa);
                A.f_out[size_t(ra) * size_t(n) + o] = xa ? -da : da;
            }
            if (rb < A.R) {
                A.x_out[size_t(rb) * size_t(n) + o] = uint8_t(xb);
                A.f_out[size_t(rb) * size_t(n) + o] = xb ? -db : db;
            }
        }
        if (Ea) atomicAdd(reinterpret_cast<unsigned long long*>(&s_e[2 * q]), (unsigned long long)Ea);
        if (Eb) atomicAdd(reinterpret_cast<unsigned long long*>(&s_e[2 * q + 1]), (unsigned long long)Eb);
        __syncthreads();
        if (tid < 32 && 32 * g + tid < A.R && s_e[tid])
            atomicAdd(reinterpret_cast<unsigned long long*>(&A.e_out[32 * g + tid]), (unsigned long long)s_e[tid]);
        __syncthreads();
    }
    if (!grid_barrier(A.bar, A.err, ++round)) return;
    for (int r = int(blockIdx.x) * kGridThreads + tid; r < A.R; r += int(gridDim.x) * kGridThreads) {
        const long long e = (long long)atomicAdd(reinterpret_cast<unsigned long long*>(&A.e_out[r]), 0ull);
        A.e_out[r] = (e + A.f0_sum) / 4;
    }
}

// A warp per bit: the word index of each neighbour (its complement's for a
// negative coupling), padded to sixteen entries with the bit itself.
__global__ void word_adjacency_kernel(const int32_t* row, const int32_t* adj, const void* w, int wbytes, const uint4* rec,
                                      int n, int wide, void* out) {
    const int lane = int(threadIdx.x & 31u);
    const int gw = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5), tw = int((gridDim.x * blockDim.x) >> 5);
    for (int i = gw; i < n; i += tw) {
        const uint4 r = rec[i];
        const int deg = int(r.y), r0 = row[i];
        const size_t o = size_t(r.x) * 16;
        for (int k = lane; k < ((deg + 15) & ~15); k += 32) {
            uint32_t e = uint32_t(i);
            if (k < deg) {
                const int v = wbytes == 1 ? int(static_cast<const int8_t*>(w)[r0 + k]) : static_cast<const int32_t*>(w)[r0 + k];
                e = uint32_t(adj[r0 + k]) + (v < 0 ? uint32_t(n) : 0u);
            }
            if (wide) static_cast<uint32_t*>(out)[o + k] = e;
            else static_cast<uint16_t*>(out)[o + k] = uint16_t(e);
        }
    }
}

}  // namespace

int64_t word_entries(const IsingPlan& p) {
    int64_t t = 0;
    for (int i = 0; i < p.n; ++i) t += (p.row[size_t(i) + 1] - p.row[size_t(i)] + 15) & ~15;
    return t;
}

int64_t word_table_bytes(const IsingPlan& p) { return word_entries(p) * p.word_bytes() + int64_t(p.n) * 16; }

qb_status upload_words(IsingPlan& p, cudaStream_t st) {
    std::vector<uint32_t> rec(size_t(p.n) * 4);
    uint32_t start = 0;   // in chunks of sixteen entries
    for (int i = 0; i < p.n; ++i) {
        const uint32_t deg = uint32_t(p.row[size_t(i) + 1] - p.row[size_t(i)]);
        rec[size_t(i) * 4] = start;
        rec[size_t(i) * 4 + 1] = deg;
        rec[size_t(i) * 4 + 2] = uint32_t(p.col.order[size_t(i)]);
        start += (deg + 15) / 16;
    }
    qb_status s;
    if ((s = upload_vec(p.d_wrec, rec, st))) return s;
    if ((s = p.d_wadj.alloc(std::max<size_t>(8, size_t(start) * 16 * size_t(p.word_bytes()))))) return s;
    const int blocks = std::max(1, std::min((p.n + 7) / 8, 148 * 8));
    word_adjacency_kernel<<<blocks, 256, 0, st>>>(p.d_row.as<int32_t>(), p.d_adj.as<int32_t>(), p.d_w.p, p.weight_bytes,
                                                  p.d_wrec.as<uint4>(), p.n, p.word_bytes() == 4 ? 1 : 0, p.d_wadj.p);
    QB_CUDA(cudaGetLastError());
    QB_CUDA(cudaStreamSynchronize(st));   // `rec` is a local
    return QB_OK;
}

int word_sms() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Read once per device: the routes' estimates ask for it several times a call.
size_t word_max_smem() {
    constexpr int kDevices = 64;
    static std::atomic<size_t> known[kDevices];
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < kDevices && known[dev].load(std::memory_order_relaxed)) return known[dev].load(std::memory_order_relaxed);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, ising_word_kernel<uint16_t>) != cudaSuccess) return 0;
    const size_t most = size_t(optin) - fa.sharedSizeBytes - sizeof(WordHead);
    if (dev < kDevices) known[dev].store(most, std::memory_order_relaxed);
    return most;
}

// Warp instructions of one sweep: a fixed part per pass of 64 proposals
// (Philox block, decisions) and one per 16 neighbours.
double word_unit_cost(int n, int64_t nnz, int np, int sweeps) {
    const double deg = n > 0 ? double(nnz) / n : 0.0;
    const double chunk = np >= 8 ? 24.0 : np == 4 ? 32.0 : 44.0;
    return double(sweeps) * (double(n) * np / 32.0) * (150.0 + chunk * std::max(1.0, deg / 16.0));
}

int word_class_passes(int n, int n_colours, int np) {
    return std::max(1, int((int64_t(n) * np + 32 * int64_t(std::max(1, n_colours)) - 1) / (32 * int64_t(std::max(1, n_colours)))));
}

// The widest unit (fewest passes of Philox lanes wasted on ragged classes)
// whose cost stays below max_cost; not wider than the replicas.
int word_pairs(const IsingPlan& p, int R, int sweeps, double max_cost) {
    int np = 16;
    while (np > 2 && np >= R) np /= 2;   // 2 np >= R still holds all replicas in one unit
    const size_t cap = word_max_smem();
    while (np > 2 && (word_item_smem(p, np) > cap || word_unit_cost(p.n, p.nnz, np, sweeps) > max_cost))
        np /= 2;
    return np;
}

void word_fill(WordItem& it, const IsingPlan& p, int np, int live, uint64_t seed0) {
    it = WordItem{};
    it.class_ptr = p.d_class_ptr.as<int32_t>();
    it.rec = p.d_wrec.as<uint4>();
    it.adj = p.d_wadj.p;
    it.seed0 = seed0;
    it.f0_sum = p.f0_sum;
    it.n = p.n;
    it.n_colours = p.col.n_colours();
    it.live = live;
    it.log2np = np == 16 ? 4 : np == 8 ? 3 : np == 4 ? 2 : 1;
    it.w0 = int32_t(p.max_w);
    it.max_deg = p.max_deg;
    it.wide = p.word_bytes() == 4 ? 1 : 0;
}

namespace {
// Teams of a CTA for a unit: split while every SM already has a unit for each
// team and either half the team would idle through an average class or the unit
// on its share of the SM stays below a quarter of the balanced makespan
// (128 mixed instances: 21.6 ms at a quarter, 26.9 at the whole; 1,024
// instances of 200 to 5,000 bits: 22.5 ms, 24.4 at a half, 28.3 at the whole)
int word_teams(size_t smem, int passes, double cost, size_t units, double total, int sms, size_t cap) {
    int t = 1;
    while (t < kMaxTeams) {
        const int t2 = 2 * t;
        if (((smem + 15) & ~size_t(15)) * size_t(t2) > cap) break;
        if (units <= size_t(t) * size_t(sms)) break;
        const bool spare = 2 * passes <= kWordThreads / 32 / t;
        const bool small = cost * t2 * sms <= 0.25 * total;
        if (!spare && !small) break;
        t = t2;
    }
    return t;
}
}  // namespace

WordWork word_pack(std::vector<WordUnit>& units) {
    std::stable_sort(units.begin(), units.end(), [](const WordUnit& a, const WordUnit& b) {
        return a.item.wide != b.item.wide ? a.item.wide < b.item.wide : a.cost > b.cost;
    });
    const int sms = word_sms();
    const size_t cap = word_max_smem();
    double total = 0.0;
    for (const WordUnit& u : units) total += u.cost;
    WordWork w;
    auto teams_of = [&](const WordUnit& u) { return word_teams(u.smem, u.passes, u.cost, units.size(), total, sms, cap); };
    for (size_t k = 0; k < units.size();) {
        const int t = teams_of(units[k]), wide = units[k].item.wide;
        WordBundle b{int32_t(w.items.size()), 0, t, 0};
        size_t need = 0;
        while (k < units.size() && b.count < t && units[k].item.wide == wide &&
               (b.count == 0 || (teams_of(units[k]) >= t && std::max(need, units[k].smem + 15) * size_t(t) <= cap))) {
            w.items.push_back(units[k].item);
            need = std::max(need, (units[k].smem + 15) & ~size_t(15));
            ++b.count;
            ++k;
        }
        b.share = int32_t(need);
        w.smem = std::max(w.smem, need * size_t(t));
        w.bundles.push_back(b);
        if (!wide) w.narrow = int(w.bundles.size());
    }
    return w;
}

namespace {
template <typename AT>
qb_status launch_width(const WordItem* items, const WordBundle* bundles, int n, size_t smem, int* counter, cudaStream_t st) {
    if (n <= 0) return QB_OK;
    QB_CUDA(allow_max_smem(ising_word_kernel<AT>));
    ising_word_kernel<AT><<<std::min(word_sms(), n), kWordThreads, sizeof(WordHead) + smem, st>>>(items, bundles, n, counter);
    QB_CUDA(cudaGetLastError());
    count_sweep(sizeof(AT) == 2 ? Sweep::kIsingWord16 : Sweep::kIsingWord32);
    return QB_OK;
}
}  // namespace

qb_status launch_ising_words(const WordWork& work, const WordItem* items, const WordBundle* bundles, int* counter,
                             cudaStream_t st) {
    QB_CUDA(cudaMemsetAsync(counter, 0, 2 * sizeof(int), st));
    qb_status s = launch_width<uint16_t>(items, bundles, work.narrow, work.smem, counter, st);
    if (s == QB_OK)
        s = launch_width<uint32_t>(items, bundles + work.narrow, int(work.bundles.size()) - work.narrow, work.smem,
                                   counter + 1, st);
    return s;
}

// More replicas than SMs: below that the few-replica sweeps have an SM for each
// replica and their shorter class step wins. QB_ISING_THREADS asks for the
// CTA-per-replica sweep's CTA size, hence for that sweep.
bool word_solve_fit(const IsingPlan& p, int R) {
    return word_sweep(p) && R > word_sms() && !std::getenv("QB_ISING_THREADS") &&
           word_item_smem(p, 2) <= word_max_smem();
}

namespace {
// The estimated microseconds of a sweep of R replicas in units of 2 np, on a
// whole device: waves of bundles, each the longer of its chain of class steps
// and its teams' instructions (2.2 a cycle), and a part of the other. A class
// step is 0.42 us and 0.07 per 16 neighbours of a bit, 0.2 where the adjacency
// exceeds the L1 cache; less in wide units on most SMs, whose lanes hold four
// stretches at once (ER(800, 0.5), 102 classes: 4.9 us a step for 149 replicas,
// 3.2 for 4,096; 300 bits of degree 24: 0.84).
double word_width_us(const IsingPlan& p, int R, int np) {
    const double nc = p.col.n_colours(), deg = double(p.nnz) / p.n;
    const int units = (R + 2 * np - 1) / (2 * np), sms = word_sms();
    const double cost = word_unit_cost(p.n, p.nnz, np, 1);
    const int t = word_teams(word_item_smem(p, np), word_class_passes(p.n, p.col.n_colours(), np), cost, size_t(units),
                             cost * units, sms, word_max_smem());
    const int bundles = (units + t - 1) / t, waves = (bundles + sms - 1) / sms;
    const bool far = p.nnz * p.word_bytes() > 160 * 1024, wide = np >= 8 && 2 * units >= sms;
    const double per = far ? (wide ? 0.115 : 0.2) : (wide ? 0.045 : 0.07);
    const double chain = nc * (0.42 + per * std::ceil(deg / 16.0));
    const double work = std::min(t, units) * cost / 4180.0;
    return waves * (std::max(chain, work) + 0.3 * std::min(chain, work));
}

// The width with the shortest estimate; near ties: the wider unit.
int word_best_pairs(const IsingPlan& p, int R, double* us) {
    int np = 2;
    *us = word_width_us(p, R, 2);
    for (int c = 4; c <= 16 && word_item_smem(p, c) <= word_max_smem(); c *= 2) {
        const double est = word_width_us(p, R, c);
        if (est < 1.02 * *us) {
            *us = est;
            np = c;
        }
    }
    return np;
}
}  // namespace

double word_solve_us(const IsingPlan& p, int R, int sweeps) {
    double us;
    word_best_pairs(p, R, &us);
    return 42.0 + sweeps * us;   // words in, fields and branches out
}

qb_status launch_word_solve(const IsingPlan& p, uint8_t* x, int32_t* f, long long* e, const double* temp, int R,
                            int sweeps, uint64_t seed0, DevBuf& tables, cudaStream_t st) {
    double us;
    const int np = word_best_pairs(p, R, &us);
    std::vector<WordUnit> units;
    for (int r0 = 0; r0 < R; r0 += 2 * np) {
        WordUnit u;
        word_fill(u.item, p, np, std::min(2 * np, R - r0), seed0 + uint64_t(r0));
        u.item.temp = temp;
        u.item.sweep1 = sweeps;
        u.item.flags = kItemInit | kItemFinal;
        u.item.e_out = e + r0;
        u.item.x_out = x + size_t(r0) * size_t(p.n);
        u.item.f_out = f + size_t(r0) * size_t(p.n);
        u.smem = word_item_smem(p, np);
        u.cost = word_unit_cost(p.n, p.nnz, np, sweeps);
        u.passes = word_class_passes(p.n, p.col.n_colours(), np);
        units.push_back(u);
    }
    const WordWork w = word_pack(units);
    const size_t ib = w.items.size() * sizeof(WordItem), bb = w.bundles.size() * sizeof(WordBundle);
    constexpr size_t kCtl = 256;
    qb_status s = tables.alloc(kCtl + ib + bb);
    if (s != QB_OK) return s;
    unsigned char* base = tables.as<unsigned char>();
    // pageable sources: the copies have taken the bytes when the calls return
    QB_CUDA(cudaMemcpyAsync(base + kCtl, w.items.data(), ib, cudaMemcpyHostToDevice, st));
    QB_CUDA(cudaMemcpyAsync(base + kCtl + ib, w.bundles.data(), bb, cudaMemcpyHostToDevice, st));
    return launch_ising_words(w, reinterpret_cast<const WordItem*>(base + kCtl),
                              reinterpret_cast<const WordBundle*>(base + kCtl + ib), reinterpret_cast<int*>(base), st);
}

// Large graphs of few classes, whose class steps can be worth a grid barrier
// (ising_route weighs it against a CTA per replica).
// The barrier's counter holds 2^32 arrivals, the pass index 2^31.
bool word_grid_fit(const IsingPlan& p, int R, int sweeps) {
    return word_sweep(p) && int64_t(p.n) * ((R + 31) / 32) < (int64_t(1) << 30) &&
           int64_t(sweeps) * p.col.n_colours() < (int64_t(1) << 24) && p.n >= 2000 * p.col.n_colours() && !std::getenv("QB_ISING_THREADS");
}

size_t word_grid_scratch(const IsingPlan& p, int R) { return 256 + size_t((R + 31) / 32) * 2 * size_t(p.n) * 4; }

qb_status launch_word_grid(const IsingPlan& p, uint8_t* x, int32_t* f, long long* e, const double* temp, int R, int sweeps,
                           uint64_t seed0, void* scratch, cudaStream_t st) {
    GridArgs A{};
    A.class_ptr = p.d_class_ptr.as<int32_t>();
    A.rec = p.d_wrec.as<uint4>();
    A.adj = p.d_wadj.p;
    A.temp = temp;
    A.bar = static_cast<unsigned*>(scratch);
    A.err = reinterpret_cast<int*>(static_cast<char*>(scratch) + 16);
    A.X = reinterpret_cast<uint32_t*>(static_cast<char*>(scratch) + 256);
    A.e_out = e;
    A.x_out = x;
    A.f_out = f;
    A.seed0 = seed0;
    A.f0_sum = p.f0_sum;
    A.n = p.n;
    A.n_colours = p.col.n_colours();
    A.sweeps = sweeps;
    A.R = R;
    A.groups = (R + 31) / 32;
    A.w0 = int32_t(p.max_w);
    A.max_deg = p.max_deg;
    QB_CUDA(cudaMemsetAsync(scratch, 0, 256, st));
    QB_CUDA(cudaMemsetAsync(e, 0, size_t(R) * 8, st));
    const void* kern = p.word_bytes() == 4 ? reinterpret_cast<const void*>(ising_grid_kernel<uint32_t>)
                                           : reinterpret_cast<const void*>(ising_grid_kernel<uint16_t>);
    void* args[] = {&A};
    QB_CUDA(cudaLaunchCooperativeKernel(kern, dim3(unsigned(word_sms())), dim3(kGridThreads), args, 0, st));
    count_sweep(p.word_bytes() == 4 ? Sweep::kIsingGrid32 : Sweep::kIsingGrid16);
    return QB_OK;
}

}  // namespace qb
