// sweep_cost.hpp — when the adjoint sweeps of several observables pay on tiles.
//
// Op by op, one kernel per gate carries every H lambda along and touches only the
// amplitudes that the gate mixes; on tiles every observable has a sweep of its own,
// a pass moves both of its states whole, and each stage of its program costs
// time.  Both are estimated in units of one read or write of a state at memory
// speed, from the compiled program on one side and the gates on the other.
//
// Fitted to Jacobians of 8 and of 60 gates of each kind on random wires, 2-16
// observables, 10-24 qubits, both precisions, with the path switched on and off:
// tiles 4-6 % rms, gates 7-8 % (22 and 24 qubits), and the dearer way is taken in
// 37 of 2924, by 24 % at most.  22 qubits complex128, 60 gates, 3
// observables, ms on tiles / op by op: DoubleExcitation (an eighth of the state
// each) 5.8 / 2.7, CSWAP 6.3 / 3.0, Toffoli 5.3 / 2.9, RX 1.8 / 9.4, IsingXX 5.2 / 8.9.
//
// No CUDA in this header: tests/cpp/sweep_cost.cpp runs the rule on the CPU.
#pragma once

#include "tile_program.hpp"

namespace plk {
namespace tile {

struct SweptOp {
    int gate;
    bool trainable;
};

// moves of a state that one observable's sweep takes
inline double sweep_moves(const TileProgram &P, bool c64) {
    double t = 4.26 * (double)P.passes.size(); // 4 of them real: lambda and H lambda, in and out
    for (const TilePass &p : P.passes) {
        const unsigned char *b = p.blob.data();
        const TileHdr &h = *reinterpret_cast<const TileHdr *>(b);
        const TileStage *S = reinterpret_cast<const TileStage *>(b + h.off_stages);
        t += (c64 ? 0.35 : 0.68) * h.nrounds;
        for (int i = 0; i < h.nstages; i++) {
            const TileStage &s = S[i];
            const bool turn = s.special == TS_CRY;
            // amplitude pairs that a controlled rotation turns
            const double active = turn ? std::ldexp((double)__builtin_popcount(s.jact), -h.R - __builtin_popcount(s.cmask)) : 0.0;
            if (c64) {
                t += 0.5 + ((s.table & 1) ? 0.35 : 0.0) + 0.2 * __builtin_popcount(s.ry) + 0.2 * active;
            } else {
                int sums_y = 0, sums_x = 0;
                for (int k = 0; k < 4; k++) {
                    sums_y += s.acc_y[k] >= 0;
                    sums_x += s.acc_x[k] >= 0;
                }
                t += ((s.table & 2) ? 0.95 : 0.0) + ((s.table & 1) ? 0.6 : 0.0) + 0.54 * __builtin_popcount(s.ry) +
                     0.36 * sums_y + 0.5 * sums_x + (turn ? 0.5 + 1.33 * active : s.special ? 1.83 : 0.0);
            }
        }
    }
    return t;
}

// full states' worth of amplitudes that a gate's kernel takes the time of
inline double gate_moves(int gate, bool c64) {
    switch (gate) {
    case PLK_GATE_PAULIX:
    case PLK_GATE_PAULIY:
    case PLK_GATE_HADAMARD: return c64 ? 1.3 : 1.2;
    case PLK_GATE_PAULIZ:
    case PLK_GATE_S:
    case PLK_GATE_T:
    case PLK_GATE_PHASESHIFT: return c64 ? 0.9 : 0.8;
    case PLK_GATE_RX:
    case PLK_GATE_RY:
    case PLK_GATE_RZ: return c64 ? 1.45 : 1.8;
    case PLK_GATE_CNOT:
    case PLK_GATE_CY:
    case PLK_GATE_SWAP: return c64 ? 0.85 : 0.77;
    case PLK_GATE_CZ: return c64 ? 0.66 : 0.5;
    case PLK_GATE_CONTROLLEDPHASESHIFT: return c64 ? 0.7 : 0.6;
    case PLK_GATE_CRX:
    case PLK_GATE_CRY:
    case PLK_GATE_CRZ: return c64 ? 0.92 : 1.03;
    case PLK_GATE_ISINGXY:
    case PLK_GATE_SINGLEEXCITATION: return c64 ? 0.98 : 1.08;
    case PLK_GATE_CSWAP:
    case PLK_GATE_TOFFOLI: return c64 ? 0.65 : 0.48;
    case PLK_GATE_DOUBLEEXCITATION: return c64 ? 0.56 : 0.43;
    case PLK_GATE_DOUBLEEXCITATIONMINUS:
    case PLK_GATE_DOUBLEEXCITATIONPLUS: return c64 ? 1.68 : 4.35;
    default: return c64 ? 1.4 : 1.82; // Ising XX, YY, ZZ, SingleExcitation+-, MultiRZ
    }
}

// One observable always: register windows, which ran it before, move the state for
// every four wires.
inline bool tiles_pay(int nobs, bool c64, const TileProgram &P, const std::vector<SweptOp> &ops) {
    if (nobs == 1) return true;
    const double move = (c64 ? 8.0 : 16.0) * std::ldexp(1.0, P.nq) / 6.78e6; // us at 6.78 TB/s
    double plain = 0.0; // with the launches, one for all states or one for each
    for (const SweptOp &op : ops)
        plain += (op.trainable ? 3.0 + 1.5 * nobs : 3.5 * (1 + nobs)) + 2.0 * (1 + nobs) * gate_moves(op.gate, c64) * move;
    return nobs * sweep_moves(P, c64) * move + 6.0 * (double)P.passes.size() <= plain;
}

} // namespace tile
} // namespace plk
