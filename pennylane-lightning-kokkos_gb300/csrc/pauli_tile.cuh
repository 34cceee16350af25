// pauli_tile.cuh — Pauli words on tiles of the state.
//
// A Pauli word pairs amplitude m with m ^ x.  One pass over the state per X
// pattern reads it as many times as there are patterns; here a pass holds tiles
// of 2^T amplitudes in shared memory, the tile's bits chosen so that as many
// patterns as possible lie inside them, and evaluates all of those words on the
// tile it has read once.  100 random words of weight 1-4 on 26 wires, 68 to 80
// patterns, take 5 or 6 passes.
#pragma once

#include <vector>

#include "pauli_plan.hpp"
#include "plk_internal.cuh"

namespace plk {

// A Pauli word P acts as P|k> = i^ny (-1)^popcount(k & z) |k ^ x>, with x the
// X/Y positions, z the Y/Z positions, ny the number of Y letters.  Terms that
// share x form one group (pauli_plan.hpp).
struct PauliTerm {
    uint64_t z;
    double cr, ci;           // c_j * i^ny
    float crh, crl, cih, cil; // the same, split for the FP32-pipe accumulation
};

// The groups that tile passes take; the others (too wide for a tile, alone in
// their pass) are left in `rest`.  `total` receives the passes' sum.
int pauli_tile_expval(plk_state s, const std::vector<PauliGroup> &groups, const std::vector<PauliTerm> &terms,
                      std::vector<PauliGroup> &rest, double &total);
// out = the taken groups' sum applied to in; `accumulate`: whether there were any
// (else nothing is written)
int pauli_tile_apply(plk_state out, plk_state in, const std::vector<PauliGroup> &groups,
                     const std::vector<PauliTerm> &terms, std::vector<PauliGroup> &rest, bool &accumulate);

} // namespace plk
