// pauli_plan.hpp — which Pauli words go to which tiles (pauli_tile.cu).
//
// No CUDA in this header: tests/cpp/pauli_plan.cpp runs the rules on the CPU.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace plk {

// the words of a sum that share the X pattern x
struct PauliGroup {
    uint64_t x;
    int first, count;
};

struct PauliTilePass {
    uint32_t bits = 0;       // state bits of the tile
    std::vector<int> groups; // indices of the groups inside
};

inline int pauli_popc(uint64_t x) { return __builtin_popcountll(x); }

// Tiles that cover the groups' X patterns: each pass starts from the widest
// pattern left, adds patterns that need the fewest more bits, and takes every
// group that lies inside.
inline void choose_passes(int nq, int T, int low, const std::vector<PauliGroup> &groups,
                          std::vector<PauliTilePass> &passes, std::vector<PauliGroup> &rest) {
    const uint64_t lowmask = (1ull << low) - 1;
    std::vector<int> left(groups.size()), fitting;
    for (size_t i = 0; i < left.size(); i++) left[i] = (int)i;
    std::stable_sort(left.begin(), left.end(), [&](int a, int b) {
        return pauli_popc(groups[a].x & ~lowmask) > pauli_popc(groups[b].x & ~lowmask);
    });
    while (!left.empty()) {
        uint64_t bits = lowmask | groups[left[0]].x;
        if (T < nq && pauli_popc(bits) > T) {
            rest.push_back(groups[left[0]]);
            left.erase(left.begin());
            continue;
        }
        fitting = left;
        for (;;) {
            int best = -1, cost = 0;
            size_t n = 0;
            for (int i : fitting) { // those inside, or too wide already, are not looked at again
                const uint64_t with = bits | groups[i].x;
                const int c = with == bits ? T + 1 : pauli_popc(with);
                if (c > T) continue;
                fitting[n++] = i;
                if (best < 0 || c < cost) {
                    best = i;
                    cost = c;
                }
            }
            fitting.resize(n);
            if (best < 0) break;
            bits |= groups[best].x;
        }
        for (int b = 0; b < nq && pauli_popc(bits) < T; b++) bits |= 1ull << b;
        PauliTilePass p;
        p.bits = (uint32_t)bits;
        size_t n = 0;
        for (int i : left) {
            if ((groups[i].x & ~bits) == 0) p.groups.push_back(i);
            else left[n++] = i;
        }
        left.resize(n);
        std::sort(p.groups.begin(), p.groups.end());
        // one group alone: a plain pass reads the state as often
        if (p.groups.size() == 1 && T < nq) rest.push_back(groups[p.groups[0]]);
        else passes.push_back(std::move(p));
    }
}

// What an application takes in us, on tiles and in plain passes: a pass without its
// words, a word on a tile, an X pattern of a plain pass (there are 32 to a pass)
// and each further word of a pattern.
//
// A tile pass reads the state and updates the output once, so its times go with the
// state's size, down to what one wave of CTAs takes: below some 20 qubits there
// are not tiles enough for the chip.  The plain kernel's go on falling, so that small
// states have it: medians by kernel at 17 to 24 qubits, sums of 2-100 words of weight
// 1-8.  24 qubits complex64: a tile pass 41 + 5.0 a word, a plain pass 19 + 13.5 a
// pattern + 37.5 a further word; 18 qubits 3.3 + 0.27 and 2.0 + 0.36 + 0.95.
// complex128: 117 + 13.5 and 90 + 55 + 114; 6.0 + 0.56 and 3.8 + 1.16 + 1.8.
struct ApplyCost {
    double pass, word, plain, group, extra;
    ApplyCost(bool c64, int nq) {
        const double s = nq >= 24 ? (double)(1ull << (nq - 24)) : 1.0 / (double)(1ull << (24 - nq));
        const double launch = 2.5; // of a pass of either kind
        auto at = [&](double least, double full) { return std::max(least, full * s); };
        pass = launch + (c64 ? at(3.3, 41) : at(6, 117));
        word = c64 ? at(0.27, 5) : at(0.55, 13.5);
        plain = launch + (c64 ? at(2, 18.6) : at(3.8, 90));
        group = c64 ? at(0.36, 13.5) : at(1.16, 55.5);
        extra = c64 ? at(0.9, 37.5) : at(1.7, 114);
    }
    // tile passes and plain passes of one sum: a second buffer and its copy
    static constexpr double both = 8;
    // finding the passes and laying out their words, for each group: 0.1-0.2 measured
    // on 100 groups, the rest because one pass seldom holds all
    static constexpr double plan = 0.3;

    double plain_time(int groups, int words) const {
        return groups ? plain * ((groups + 31) / 32) + group * groups + extra * (words - groups) : 0.0;
    }
    // Is a search for passes worth its time?  All words in one pass are the best it can find.
    bool worth_a_look(const std::vector<PauliGroup> &all) const {
        int words = 0;
        for (const PauliGroup &g : all) words += g.count;
        return pass + word * words + plan * (double)all.size() < plain_time((int)all.size(), words);
    }
};

// Application: the passes with most words on tiles, the others plain, whichever
// split is cheapest.
inline void keep_worthwhile(const ApplyCost &c, const std::vector<PauliGroup> &groups,
                            std::vector<PauliTilePass> &passes, std::vector<PauliGroup> &rest) {
    auto words = [&](const PauliTilePass &p) {
        int n = 0;
        for (int gi : p.groups) n += groups[gi].count;
        return n;
    };
    std::stable_sort(passes.begin(), passes.end(),
                     [&](const PauliTilePass &x, const PauliTilePass &y) { return words(x) > words(y); });
    int plain_groups = (int)rest.size(), plain_words = 0;
    for (const PauliGroup &g : rest) plain_words += g.count;
    double on_tiles = 0.0, least = 0.0;
    for (const PauliTilePass &p : passes) on_tiles += c.pass + c.word * words(p);
    size_t best = passes.size();
    for (size_t k = passes.size() + 1; k-- > 0;) {
        if (k < passes.size()) {
            on_tiles -= c.pass + c.word * words(passes[k]);
            plain_groups += (int)passes[k].groups.size();
            plain_words += words(passes[k]);
        }
        const double cost = (k ? on_tiles : 0.0) + c.plain_time(plain_groups, plain_words) +
                            (k && plain_groups ? c.both : 0.0);
        if (k == passes.size() || cost < least) {
            least = cost;
            best = k;
        }
    }
    for (size_t k = best; k < passes.size(); k++)
        for (int gi : passes[k].groups) rest.push_back(groups[gi]);
    passes.resize(best);
}

} // namespace plk
