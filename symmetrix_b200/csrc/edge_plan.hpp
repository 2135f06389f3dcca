// What the host goes by while it does not know a structure's number of edges (host only, no CUDA).
#pragma once

#include <algorithm>

namespace smx {

// Are an evaluation's kernels launched overlapped (Launcher::overlap)? Yes while launch gaps are what it loses; beyond, the
// successor's CTAs, resident early, cost the running kernel L1 and slots. Call time without / with overlap, by edges x num_LM x K:
// float64, 128 channels, fcc: 1.9M 1.09, 5.8M 1.04, 9.6M 1.01, 13M 0.99, 19M 0.99, 29M 0.97, 82M 0.97; water 5.4M 1.07, 10M 1.04,
// 18M 1.01, 28M 0.99, 83M 0.98; 64 channels, L_max = 0: 10M 1.02, 18M 1.01, 28M 0.99. float32, whose kernels are half as long: fcc
// 9.6M 1.04, 24M 1.04, 29M 1.03, 40M 0.98, 55M 1.00; water 18M 1.03, 28M 1.05, 42M 1.04, 60M 1.02; L_max = 0 28M 1.02. Two kernels
// are left out where they lose by it (Evaluator::run_gemms, launch_tp).
inline bool overlap_pays(long edges, int num_LM, int K, bool float64) {
    return static_cast<double>(edges) * num_LM * K <= (float64 ? 2e7 : 3e7);
}

// Edges to expect of a structure that is evaluated in one call, where the number is known only afterwards. Launches, work items
// and scratch are sized by it, so it follows the structures and not the arrays: those keep the size of the largest structure a
// handle has seen, and a molecule evaluated after a box of 4,000 atoms is a molecule.
class EdgePlan {
public:
    static constexpr long kFreeEdges = 16384;         // at least 64 per atom within this: no molecule or unit cell runs out of room
    static constexpr double kGuessBytes = 256e6;      // memory that may be asked for on a guess

    // By the densest of the recent structures, fading by a tenth a call: sparse and dense ones may alternate without starting again.
    long likely(long atoms) const { return static_cast<long>(static_cast<double>(atoms) * per_atom); }
    // Edges to make room for (an eighth more than likely), or -1: count them first, where the guess would take much memory that is
    // not there yet (`allocated`: edges the arrays hold). Counting first costs 30 us in 2.2 ms (207 atoms, K = 256, L_max = 2).
    long room(long atoms, double bytes_per_edge, long allocated) const {
        const long l = likely(atoms), r = l + l / 8, roomy = std::max(r, std::min(64 * atoms, kFreeEdges));
        for (long want : {roomy, r})
            if (static_cast<double>(want) * bytes_per_edge <= kGuessBytes) return want;
        return allocated >= l + l / 64 ? std::min(r, allocated) : -1;
    }
    void seen(long atoms, long edges) {
        if (atoms <= 0) return;
        const double now = static_cast<double>(edges) / static_cast<double>(atoms);
        per_atom = any ? std::max(now, 0.9 * per_atom) : now;
        any = true;
    }

private:
    double per_atom = 64.0;       // until a structure has been seen
    bool any = false;
};

}  // namespace smx
