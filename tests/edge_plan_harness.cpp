// Prints what csrc/edge_plan.hpp decides after a sequence of structures: argv is <num_LM> <K> <bytes per edge> and then
// triples <atoms> <edges> <allocated>; for each, before it is seen: likely, room and whether the launches overlap.
#include <cstdio>
#include <cstdlib>

#include "edge_plan.hpp"

int main(int argc, char** argv) {
    const int num_LM = std::atoi(argv[1]), K = std::atoi(argv[2]);
    const double bytes = std::atof(argv[3]);
    smx::EdgePlan plan;
    for (int q = 4; q + 2 < argc; q += 3) {
        const long atoms = std::atol(argv[q]), edges = std::atol(argv[q + 1]), allocated = std::atol(argv[q + 2]);
        const long room = plan.room(atoms, bytes, allocated);
        std::printf("%ld %ld %d\n", plan.likely(atoms), room, smx::overlap_pays(room < 0 ? edges : room, num_LM, K, true) ? 1 : 0);
        plan.seen(atoms, edges);
    }
}
