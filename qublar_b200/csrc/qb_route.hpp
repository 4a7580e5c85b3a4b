// Which sweep a single integer solve takes. All give the same branches; the
// choice is the shortest estimated time, from times measured on a B200.
#pragma once

#include "qb_internal.hpp"

namespace qb {

// Large graphs of one coupling size on the whole device (qb_word.cu); few
// replicas and dense graphs (qb_replica.cu); many replicas of one coupling
// size (qb_word.cu); otherwise a CTA per replica with its fields (qb_kernels.cu).
enum class IsingRoute { kGrid, kReplicas, kWords, kFields };

// t_max: the schedule's largest temperature; traced: per-sweep energies wanted
// (the word and the grid sweep record none).
IsingRoute ising_route(const IsingPlan& p, int R, int sweeps, double t_max, bool traced);

}  // namespace qb
