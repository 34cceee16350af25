// The rules that send the words of an applied Pauli sum to tiles or to the plain
// kernel (csrc/pauli_plan.hpp), for tests/test_pauli_plan_cpu.py.
#include "pauli_plan.hpp"

using namespace plk;

static std::vector<PauliGroup> make(int n, const uint64_t *x, const int *count) {
    std::vector<PauliGroup> g;
    for (int i = 0, at = 0; i < n; at += count[i], i++) g.push_back({x[i], at, count[i]});
    return g;
}

// pass_of[i]: the pass that takes group i, -1 for none; returns the number of passes
extern "C" int plan_passes(int nq, int T, int low, int n, const uint64_t *x, const int *count, int *pass_of,
                           uint32_t *bits) {
    const std::vector<PauliGroup> g = make(n, x, count);
    std::vector<PauliTilePass> passes;
    std::vector<PauliGroup> rest;
    choose_passes(nq, T, low, g, passes, rest);
    for (int i = 0; i < n; i++) pass_of[i] = -1;
    size_t taken = rest.size();
    for (size_t p = 0; p < passes.size(); p++) {
        bits[p] = passes[p].bits;
        taken += passes[p].groups.size();
        for (int i : passes[p].groups) pass_of[i] = (int)p;
    }
    return taken == g.size() ? (int)passes.size() : -1;
}

// words on tiles of an application
extern "C" int plan_words_on_tiles(int nq, int c64, int n, const uint64_t *x, const int *count) {
    const std::vector<PauliGroup> g = make(n, x, count);
    const ApplyCost cost(c64 != 0, nq);
    if (!cost.worth_a_look(g)) return 0;
    std::vector<PauliTilePass> passes;
    std::vector<PauliGroup> rest;
    choose_passes(nq, 12, c64 ? 3 : 2, g, passes, rest);
    keep_worthwhile(cost, g, passes, rest);
    int words = 0;
    for (const PauliTilePass &p : passes)
        for (int i : p.groups) words += g[i].count;
    return words;
}
