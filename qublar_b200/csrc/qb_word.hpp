// Integer Ising graphs of one coupling size (every |w_ij| = w0: unweighted
// and +-1 Max-Cut): replicas as the bits of a word, fields counted from the
// neighbours' words when a bit is visited.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "qb_internal.hpp"

namespace qb {

// The largest degree the per-sweep threshold table serves.
constexpr int kWordMaxDegree = 1024;
constexpr int kWordThreads = 768;

// One unit of work: G = 2 NP replicas of one instance (word bit p is replica
// 2p, bit p + NP replica 2p + 1) over sweeps [sweep0, sweep1).
struct WordItem {
    const int32_t* class_ptr;   // n_colours + 1
    const uint4* rec;           // per bit {first entry / 16, degree, original bit, 0}
    const void* adj;            // rows of word indices (uint16 or uint32): j, or n + j (j's complement)
                                // for w_ij < 0; padded to sixteen entries with the bit itself
    const double* temp;
    void* state;                // n words of G bits kept between slices (kItemKeep; no kItemInit)
    long long* e_out;           // live tracked energies (kItemFinal)
    uint8_t* x_out;             // live x n, original order (kItemFinal)
    int32_t* f_out;             // live x n
    uint64_t seed0;             // seed of the unit's first replica (an even one of its solve)
    long long f0_sum;           // sum of the fields of x = 0 (= -2 sum_e w)
    int32_t n;
    int32_t n_colours;
    int32_t log2np;             // 1 .. 4
    int32_t live;               // replicas of the unit that exist (1 .. G)
    int32_t sweep0;
    int32_t sweep1;
    int32_t flags;              // kItemInit, kItemFinal, kItemKeep (qb_batch.hpp)
    int32_t w0;
    int32_t max_deg;
    int32_t wide;               // 1: uint32 adjacency
};

// Items [first, first + count) run side by side on the CTA's `teams` teams
// (1, 2, 4 or 8 of kWordThreads / teams threads each).
struct WordBundle {
    int32_t first;
    int32_t count;
    int32_t teams;
    int32_t share;   // shared memory of one team, bytes
};

// Whether a plan has the word sweep's form: one coupling size and degrees its
// threshold table holds.
inline bool word_sweep(const IsingPlan& p) { return p.one_size && p.max_deg <= kWordMaxDegree; }

// Bytes a unit takes of its team's shared memory: thresholds, class
// boundaries, words and complements (whole bytes).
inline size_t word_item_smem(const IsingPlan& p, int np) {
    return (2 * size_t(p.max_deg) + 1) * 8 + (size_t(p.col.n_colours()) + 1) * 4 +
           2 * size_t(p.n) * size_t(np > 4 ? np / 4 : 1);
}

// The word tables of a plan: their device bytes, and their upload (after the
// plan's own arrays).
int64_t word_table_bytes(const IsingPlan& p);
qb_status upload_words(IsingPlan& p, cudaStream_t st);

size_t word_max_smem();
int word_sms();

// One unit before it is placed: what its placement needs, and its item.
struct WordUnit {
    WordItem item;
    double cost;      // relative device time on one whole SM
    int passes;       // warp passes of an average class
    size_t smem;      // word_item_smem
};
double word_unit_cost(int n, int64_t nnz, int np, int sweeps);
int word_class_passes(int n, int n_colours, int np);
// Pairs per unit for R replicas of an instance, given the cost a unit may have.
int word_pairs(const IsingPlan& p, int R, int sweeps, double max_cost);
// The launch tables of a set of units: items and bundles, those with 16-bit
// adjacency first, and the dynamic shared memory (what is not asked for serves
// as L1 cache for the adjacency).
struct WordWork {
    std::vector<WordItem> items;
    std::vector<WordBundle> bundles;
    int narrow = 0;   // bundles with 16-bit adjacency
    size_t smem = 0;
};
// Orders the units largest first and packs them into bundles.
WordWork word_pack(std::vector<WordUnit>& units);
// Fills a unit's item from a plan (replicas r0 .. r0 + live of the solve).
void word_fill(WordItem& it, const IsingPlan& p, int np, int live, uint64_t seed0);
// Runs the work (its tables on the device); counter: two device ints.
qb_status launch_ising_words(const WordWork& work, const WordItem* items, const WordBundle* bundles, int* counter,
                             cudaStream_t st);

// A single solve of a large graph on the whole device (scratch: word_grid_scratch
// bytes, the barrier's timeout flag at +16).
bool word_grid_fit(const IsingPlan& p, int R, int sweeps);
size_t word_grid_scratch(const IsingPlan& p, int R);
qb_status launch_word_grid(const IsingPlan& p, uint8_t* x, int32_t* f, long long* e, const double* temp, int R, int sweeps,
                           uint64_t seed0, void* scratch, cudaStream_t st);
// A single solve of R replicas as word units: whether the route serves it, the
// estimated time of the solve in microseconds, and the launch (tables: one
// device allocation, kept until the stream's work is done; x, f, e: R x n, R x
// n, R).
bool word_solve_fit(const IsingPlan& p, int R);
double word_solve_us(const IsingPlan& p, int R, int sweeps);
qb_status launch_word_solve(const IsingPlan& p, uint8_t* x, int32_t* f, long long* e, const double* temp, int R,
                            int sweeps, uint64_t seed0, DevBuf& tables, cudaStream_t st);

}  // namespace qb
