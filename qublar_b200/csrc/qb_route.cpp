// The route of a single integer solve: estimates of a solve's microseconds on a
// B200 for each kernel that can serve it, fitted to measured kernel times over
// 25 to 60,000 bits, degrees 3 to 450 and 149 to 8,192 replicas (497 points; the
// choice costs 0.5 % over the best kernel on average, at most 30 %; the wrong
// kernel up to 8 times).
#include <algorithm>
#include <cmath>

#include "qb_kernels.hpp"
#include "qb_route.hpp"
#include "qb_word.hpp"

namespace qb {

namespace {

// The CTA-per-replica sweep with more replicas than SMs (128-thread CTAs, up to
// twelve an SM): a wave's class step takes 0.55 us and, per bit of it, a few ns
// that grow with its rows (an accepted flip's row is added by a warp); many
// replicas are bound by the SM's instructions instead, 45 ns a class step and
// about 1 to 5 a bit for each.
double fields_solve_us(const IsingPlan& p, int R, int sweeps) {
    const double nc = p.col.n_colours(), bits = p.n / nc, deg = double(p.nnz) / p.n, sms = word_sms();
    const double per_bit = deg < 16.0    ? 0.003 + 0.00035 * deg
                           : deg <= 110.0 ? 0.009 + 0.0003 * std::min(deg, 90.0)
                                          : 0.026 + 0.0002 * std::max(0.0, deg - 170.0);
    const double step = 0.55 + per_bit * (std::min(bits, 256.0) + 2.0 * std::max(0.0, bits - 256.0));
    const double busy = (0.045 + bits * (0.00085 + 0.00004 * std::min(deg, 100.0))) * R / sms;
    const double fit = std::min(12.0, std::max(1.0, std::floor(160.0 * 1024 / (5.0 * p.n + 1024))));
    const double chain = std::ceil(R / (sms * fit)) * step;
    return 8.0 + sweeps * nc * (std::max(chain, busy) + 0.2 * std::min(step, std::max(0.0, busy - 0.5 * step)));
}

// Whether the whole-device sweep's class step is the shorter one for at most one
// replica per SM. It takes 3.7 us (the grid barrier and one round of the
// device's warps over two bits each) and 1.6 for each further round; a class of
// the few-replica sweep with its adjacency on chip 0.35 us and about 1 ns a bit
// (1.45 without helper CTAs); of the CTA-per-replica sweep 2 ns a bit, 1.6 where
// the L1 cache holds the adjacency. 40 sweeps, 16 and 148 replicas: 4,096 bits in
// 2 classes 0.30 and 0.45 ms grid, 0.26 and 0.26 CTA per replica; 20,000 bits in
// 4, 0.57 and 1.1 against 1.6.
bool grid_pays(const IsingPlan& p, int R, bool few) {
    const double nc = p.col.n_colours(), bits = p.n / nc, sms = word_sms();
    const double x = std::ceil(bits / 2.0) * ((R + 31) / 32) / (32.0 * sms);
    const double grid = 3.7 + 0.2 * x + 1.6 * (std::ceil(x) - 1.0);
    const double cta = few && replica_csr_fit(p) ? 0.35 + (2 * R <= sms ? 0.00105 : 0.00145) * bits
                       : (p.nnz * (4 + p.weight_bytes) < 96 * 1024 ? 0.0016 : 0.0020) * bits;
    return grid < 1.05 * cta;
}

}  // namespace

IsingRoute ising_route(const IsingPlan& p, int R, int sweeps, double t_max, bool traced) {
    const bool words = !traced && word_solve_fit(p, R);
    const bool grid = !traced && !words && word_grid_fit(p, R, sweeps);
    const bool few = replica_solve_fit(p, R, t_max);
    // at most one replica per SM: the class chain's length decides, and of the
    // others the few-replica sweeps have the shorter one wherever they fit
    if (R <= word_sms()) return grid && grid_pays(p, R, few) ? IsingRoute::kGrid : few ? IsingRoute::kReplicas : IsingRoute::kFields;
    if (grid) return IsingRoute::kGrid;   // words of a graph too large for a CTA's shared memory
    // more replicas: the dense kernel keeps a CTA, and of it one warp, per
    // replica; the word sweep has the fewer instructions but a long class step
    // on long rows
    IsingRoute best = IsingRoute::kFields;
    double us = fields_solve_us(p, R, sweeps);
    if (words) {
        const double w = word_solve_us(p, R, sweeps);
        if (w < us) {
            best = IsingRoute::kWords;
            us = w;
        }
    }
    if (few && dense_solve_us(p, R, sweeps) < us) best = IsingRoute::kReplicas;
    return best;
}

}  // namespace qb
