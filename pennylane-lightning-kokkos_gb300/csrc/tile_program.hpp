// tile_program.hpp — host side of the tile sweeps: an op list becomes a few
// passes over the state, each a program that a CTA runs on tiles of 2^T
// amplitudes held in shared memory (tile_kernels.cuh).
//
// Lowering.  Every named gate is written as rotations [[c, -s], [s, c]] on one
// bit (with controls), diagonal phases, and index maps (CNOT, X, SWAP):
//   RX = S^dag RY S, IsingXX = CX (RX x 1) CX, IsingYY = S S (XX) S^dag S^dag,
//   SingleExcitation = CX(a,b) controlled-RY(a | b = 1) CX(a,b), and so on;
// runs of one-wire gates on one wire are multiplied and split as
// diag RY diag (|s| <= c: a half turn is taken out as an X).  complex64 runs the
// rotation as three shears in place; complex128 as [[1, -t], [t, 1]], t = s / c,
// whose factor c goes into the next phase table (two double-float products per
// amplitude pair instead of three).  Index maps move no data: a tile keeps the linear map over
// GF(2) from logical index to shared-memory slot and composes CNOTs into it; a
// CNOT whose control lies outside the tile flips a constant of that map.
//
// Gradients.  Im <h|G|v> of every gate reduces to a few sums over the tile's
// amplitudes: Im <h|X|v> and Im <h|Y|v> on a rotated bit, and signed sums
// (Walsh functions of register bits) of c_j = Im(conj h_j v_j) for diagonal
// generators.  With a run's gates multiplied, the generators inside the run
// are rotated to its frame: real combinations of the three sums.  An
// accumulator holds one sum; the Jacobian is a sparse combination of them.
//
// Scheduling.  A list schedule over the dependency graph (two ops that are
// both diagonal, or both flips, on every wire they share commute) fills a tile
// with all ops that fit its bits, then splits them into rounds of R register
// bits: a thread holds 2^R amplitudes in registers and runs the round's stages
// on them (a phase table, then rotations of the register bits, then at most one
// step that needs the state index).  The first round reads the state and the
// last one writes it, in between a round hands its amplitudes to the next
// through shared memory, each thread writing to the slots it read.
//
// No CUDA in this header: tests/cpp/tile_emulator.cpp runs the same programs
// on the CPU.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "plk_gb300.h"

namespace plk {
namespace tile {

constexpr int kMaxRegBits = 4;     // register bits of a round (R), at most
constexpr int kMaxAmps = 16;
constexpr int kMaxTileBits = 12;   // largest tiles of the launch shapes; slot offsets in bytes fit 16 bits
constexpr int kMaxAcc = 128;       // accumulators per pass
constexpr int kMaxUnits = 192;     // ops per pass
constexpr double kTiny = 1e-15;

// ------------------------------------------------------ device structures --
enum SpecialKind : uint8_t { TS_NONE = 0, TS_CRY = 1, TS_DIAG = 2, TS_PAR = 3 };

// Order within a stage: sums of the table, table, rotations by ascending bit,
// special step.
struct alignas(16) TileStage { // 144 bytes
    float rot[4][4]; // bit b: complex64 the shears t, s as t.hi t.lo s.hi s.lo; complex128 t = s / c as t.hi t.lo
    int16_t acc_y[4], acc_zb[4]; // accumulators of Im <h|Y|v> by bit, of the Walsh sums when all are of single bits (-1: none)
    uint8_t ry;      // bits that turn
    uint8_t table;   // bit 0: sums wanted (zsel), bit 1: phases to apply
    uint8_t special; // SpecialKind
    uint8_t sums;    // bit 0: some acc_y, bit 1: some acc_x
    uint16_t tab;    // first table entry
    uint16_t zsel;   // Walsh functions wanted (bit m: mask m over register bits)
    int16_t acc_z;   // accumulator of the lowest set bit of zsel, the others follow
    // special step
    uint8_t bit, K;  // CRY: register bit; DIAG: bits of the table index
    uint16_t jact;   // CRY: amplitudes whose register bits satisfy the controls
    uint16_t stab;   // DIAG, PAR: first table entry
    uint32_t cmask, cval; // CRY: control bits of the state index; PAR: mask; DIAG: state bit of table bit i in bits 5i..
    uint32_t gtab;   // DIAG: generator values (float), first entry
    int16_t sacc;    // accumulator of the special step (-1: none)
    uint16_t pad;
    float coef[4];   // CRY: c.hi c.lo s.hi s.lo
    int16_t acc_x[4]; // accumulators of Im <h|X|v>
    uint32_t pad2[2];
};
static_assert(sizeof(TileStage) == 144, "stage size");
static_assert(offsetof(TileStage, ry) == 80 && offsetof(TileStage, stab) == 94, "ry .. stab are read as 16 bytes");
static_assert(offsetof(TileStage, acc_zb) == offsetof(TileStage, acc_y) + 8, "one list of eight");

struct alignas(16) TileRound { // 128 bytes
    uint16_t lo[32]; // byte offset in the tile of lane bits,
    uint16_t hi[16]; // of thread bits above the lane,
    uint16_t rcol[kMaxRegBits]; // of register bits (combined by exclusive or)
    uint16_t xorc;
    uint16_t stage0, nstages;
    uint16_t ev0, nev; // flips of the map's constant before the round
    uint16_t idx;      // state index of (thread, register) for special steps (0xffff: none)
    uint16_t pad[6];
};
static_assert(sizeof(TileRound) == 128, "round size");
static_assert(offsetof(TileRound, rcol) == 96 && offsetof(TileRound, ev0) == 110, "rcol .. ev0 are read as 16 bytes");

struct TileEvent { // when state bit `bit` of the tile's base is set, the map's constant is flipped
    uint16_t mask, bit; // byte offset
    uint32_t gmask;     // state index (events before the first and after the last round)
};

struct alignas(16) TileIndex { // state index relative to the tile's base (combined by exclusive or)
    uint32_t lo[32], hi[16], r[kMaxRegBits];
    uint32_t c, pad[3];
};

struct alignas(16) TileHdr {
    int32_t T, R, nq, nrounds, nstages, nacc, acc0;
    uint32_t off_rounds, off_stages, off_events, off_index, off_tab, bytes;
    int32_t nev, ev_store0; // events from ev_store0 on belong to the store
    uint32_t load_idx, store_idx; // where the first round reads, the last writes
    uint8_t gpos[16]; // state bit of tile bit i (ascending)
    uint32_t pad[3];
};
static_assert(sizeof(TileHdr) % 16 == 0, "header size");

// one pass over the state
struct TilePass {
    std::vector<unsigned char> blob; // TileHdr first, 16-byte aligned size
};

struct JacTerm {
    int32_t slot, acc;
    double coef;
    int32_t ref = -1; // symbolic programs: the coefficient is coef * refs[ref]
};

struct TileProgram {
    int nq = 0, T = 0, R = 0;
    bool bwd = false;
    int nacc = 0;
    std::vector<TilePass> passes;
    std::vector<JacTerm> jac;
};

// Every index that a kernel follows, checked before the first launch.
inline bool check_pass(const TilePass &p, int nq, int amp_bytes, int nacc_all) {
    const unsigned char *b = p.blob.data();
    const TileHdr &h = *reinterpret_cast<const TileHdr *>(b);
    if (p.blob.size() != h.bytes || h.nq != nq || h.R < 1 || h.R > kMaxRegBits || h.T < h.R || h.T > nq ||
        h.T > kMaxTileBits || h.nrounds < 1)
        return false;
    if (h.acc0 < 0 || h.nacc < 0 || h.nacc > 2 * kMaxAcc || h.acc0 + h.nacc > nacc_all) return false;
    const uint32_t tile = (uint32_t)amp_bytes << h.T;
    if (tile > 65536) return false;
    uint32_t bits = 0;
    for (int k = 0; k < h.T; k++) {
        if (h.gpos[k] >= nq || (k && h.gpos[k] <= h.gpos[k - 1])) return false;
        bits |= 1u << h.gpos[k];
    }
    const TileRound *R = reinterpret_cast<const TileRound *>(b + h.off_rounds);
    const TileStage *S = reinterpret_cast<const TileStage *>(b + h.off_stages);
    const TileEvent *E = reinterpret_cast<const TileEvent *>(b + h.off_events);
    const TileIndex *X = reinterpret_cast<const TileIndex *>(b + h.off_index);
    const size_t nidx = (h.off_tab - h.off_index) / sizeof(TileIndex), ntab = (h.bytes - h.off_tab) / amp_bytes;
    if (h.load_idx >= nidx || h.store_idx >= nidx || h.ev_store0 > h.nev) return false;
    for (size_t i = 0; i < nidx; i++) {
        uint32_t all = X[i].c;
        for (uint32_t x : X[i].lo) all |= x;
        for (uint32_t x : X[i].hi) all |= x;
        for (int k = 0; k < h.R; k++) all |= X[i].r[k];
        if (all & ~bits) return false;
    }
    for (int k = 0; k < h.nev; k++)
        if (E[k].bit >= nq || E[k].mask >= tile || E[k].mask % amp_bytes || (E[k].gmask & ~bits)) return false;
    for (int r = 0; r < h.nrounds; r++) {
        uint32_t all = R[r].xorc;
        for (uint16_t x : R[r].lo) all |= x;
        for (uint16_t x : R[r].hi) all |= x;
        for (int k = 0; k < h.R; k++) all |= R[r].rcol[k];
        if (all >= tile || all % amp_bytes || R[r].stage0 + R[r].nstages > h.nstages || R[r].ev0 + R[r].nev > h.nev)
            return false;
        if (R[r].idx != 0xffff && R[r].idx >= nidx) return false;
        for (int k = 0; k < R[r].nstages; k++) {
            const TileStage &t = S[R[r].stage0 + k];
            for (int i = 0; i < 4; i++)
                if (t.acc_y[i] >= h.nacc || t.acc_x[i] >= h.nacc || t.acc_zb[i] >= h.nacc) return false;
            if (t.ry >> h.R) return false;
            if ((t.table & 2) && t.tab + (size_t)(1 << h.R) > ntab) return false;
            if ((t.table & 1) && (t.acc_z < 0 || t.acc_z + __builtin_popcount(t.zsel) > h.nacc)) return false;
            const size_t len = t.special == TS_PAR ? 2 : t.special == TS_DIAG ? 1u << t.K : 0;
            if (t.special > TS_PAR || t.bit >= h.R || t.K > 3 || t.stab + len > ntab || t.sacc >= h.nacc) return false;
            if ((t.special >= TS_DIAG || (t.special == TS_CRY && t.cmask)) && R[r].idx == 0xffff) return false;
            if (t.special == TS_DIAG && t.sacc >= 0 && (t.gtab + len) * sizeof(float) > h.bytes - h.off_tab) return false;
        }
    }
    return true;
}

// --------------------------------------------------------------- lowering --
using cplx = std::complex<double>;

struct Grad {
    int slot;
    double g[4]; // U1: coefficients of I, X, Y, Z; CRY: g[2]; PAR: g[3]
    std::vector<double> table; // DIAG: generator diagonal (table index order)
    double coef = 1.0;         // DIAG
};

enum PrimKind { P_U1, P_DIAG, P_PAR, P_CRY, P_CX, P_X, P_SWAP };

// ---- symbolic programs -----------------------------------------------------
// A batch compiles its circuits once, for any parameters: the program's numbers
// (tables, rotations, coefficients) are left open and listed here, and a kernel
// fills them in for each run (batch_tile.cu).  A gate's entries are
// A0 + A1 cos(t/2) + A2 sin(t/2) + A3 cos(t) + A4 sin(t): `basis` is the offset
// of its five coefficients per entry.
enum GateForm : uint8_t { GF_DIAG = 0, GF_RY = 1, GF_OTHER = 2 };
enum RunType : uint8_t { RT_DIAG = 0, RT_RIGHT = 1, RT_LEFT = 2, RT_GENERAL = 3 };

struct SymGate { // one gate of a run of one-wire gates
    int32_t basis, pidx; // pidx -1: constant
    int32_t next;        // the run's next gate, -1 at its end
    int32_t form;
    double g[4];         // generator: coefficients of I, X, Y, Z
    int32_t ref[4];      // refs of its I, X, Y, Z coefficients in the frame of the run's sums (-1: not wanted)
};
struct SymRun { // diag(b) RY(c, s) diag(a), or the diagonal itself
    int32_t head, type;
    int32_t pool_a, pool_b; // two entries each; RT_DIAG: pool_a
};
struct SymEval { // entries of another gate
    int32_t basis, pidx, n, pool;
};
struct SymFactor { // part of a table: pool[k], k = register bits reg[0..K) of j; K = -1: the parity of j & mask
    int32_t pool;
    int8_t K;
    uint8_t reg[3];
    uint8_t mask, pad[3];
};
struct SymTable { // a phase table: the product of its factors
    int32_t pass;
    uint32_t off; // byte offset in the pass's blob
    int32_t first, count;
};
struct SymPatch { // kind 0: rotation of run `src`; 1: c, s from pool; 2: n entries from pool
    int32_t pass;
    uint32_t off;
    int32_t kind, src, n;
};
struct Symbols {
    std::vector<SymGate> gates;
    std::vector<SymRun> runs;
    std::vector<SymEval> evals;
    std::vector<SymFactor> factors;
    std::vector<SymTable> tables;
    std::vector<SymPatch> patches;
    int npool = 0, nrefs = 0;
};

struct Prim {
    int kind = P_U1;
    int sbasis = -1, spidx = -1;      // symbolic: coefficients of the entries
    int shead = -1, stail = -1;       // symbolic U1: its gates
    int t = 0, t2 = 0;          // target state bits
    uint32_t cmask = 0, cval = 0; // CRY controls; CX: control bit mask
    double c = 1, s = 0;        // CRY
    cplx m[4] = {1, 0, 0, 1};   // U1
    int K = 0;                  // DIAG
    int db[4] = {0, 0, 0, 0};   // DIAG: state bit of table index bit i
    cplx d[8];                  // DIAG: 2^K, PAR: 2
    uint32_t pmask = 0;         // PAR
    std::vector<Grad> grads;
};

struct Lowered {
    std::vector<Prim> v;

    void u1(int b, cplx a, cplx bb, cplx c, cplx d) {
        Prim p;
        p.kind = P_U1;
        p.t = b;
        p.m[0] = a;
        p.m[1] = bb;
        p.m[2] = c;
        p.m[3] = d;
        v.push_back(p);
    }
    void diag1(int b, cplx e0, cplx e1) { u1(b, e0, 0, 0, e1); }
    void cx(int c, int t) {
        Prim p;
        p.kind = P_CX;
        p.t = t;
        p.cmask = 1u << c;
        v.push_back(p);
    }
    void x(int t) {
        Prim p;
        p.kind = P_X;
        p.t = t;
        v.push_back(p);
    }
    void swap(int a, int b) {
        Prim p;
        p.kind = P_SWAP;
        p.t = a;
        p.t2 = b;
        v.push_back(p);
    }
    void cry(int t, uint32_t cm, uint32_t cv, double c, double s) {
        Prim p;
        p.kind = P_CRY;
        p.t = t;
        p.cmask = cm;
        p.cval = cv;
        p.c = c;
        p.s = s;
        v.push_back(p);
    }
    // table index bit i <-> state bit bits[i]
    void diag(std::initializer_list<int> bits, std::initializer_list<cplx> d) {
        Prim p;
        p.kind = P_DIAG;
        for (int b : bits) p.db[p.K++] = b;
        std::copy(d.begin(), d.end(), p.d);
        v.push_back(p);
    }
    void grad_u1(int slot, double gi, double gx, double gy, double gz) {
        v.back().grads.push_back(Grad{slot, {gi, gx, gy, gz}, {}, 1.0});
    }
    void grad_diag(int slot, double coef, std::vector<double> table) {
        v.back().grads.push_back(Grad{slot, {0, 0, 0, 0}, std::move(table), coef});
    }
};

inline cplx expi(double t) { return cplx(std::cos(t), std::sin(t)); }

// Lowers one op (applied with its adjoint flag) to primitives in application
// order; slot >= 0: the Jacobian slot of its parameter.  Jacobian terms are
// written for Jac = Im <h|G|v> of a gate exp(-i t G / 2).  False: not a gate of
// this path.
inline bool lower_op(const plk_op &op, int nq, int slot, Lowered &L) {
    const bool inv = op.adjoint != 0;
    const double th0 = op.num_params > 0 && op.params ? op.params[0] : 0.0;
    const double th = inv ? -th0 : th0;
    const double sg = inv ? -1.0 : 1.0; // d(applied angle) / d(parameter)
    const double c = std::cos(th / 2), s = std::sin(th / 2);
    const cplx i1(0, 1);
    int b[4] = {0, 0, 0, 0};
    if (op.gate != PLK_GATE_MULTIRZ) {
        if (op.num_wires < 1 || op.num_wires > 4) return false;
        for (int j = 0; j < op.num_wires; j++) b[j] = nq - 1 - (int)op.wires[j];
    }
    auto S = [&](int t) { L.diag1(t, 1, i1); };
    auto Sd = [&](int t) { L.diag1(t, 1, -i1); };
    auto bit = [](int x) { return 1u << x; };
    auto grad_cry = [&](double k) {
        if (slot >= 0) L.v.back().grads.push_back(Grad{slot, {0, 0, k, 0}, {}, 1.0});
    };
    const double r = std::sqrt(0.5);
    switch (op.gate) {
    case PLK_GATE_IDENTITY: return true;
    case PLK_GATE_PAULIX: L.x(b[0]); return true;
    case PLK_GATE_PAULIY: L.diag1(b[0], i1, -i1); L.x(b[0]); return true;
    case PLK_GATE_PAULIZ: L.diag1(b[0], 1, -1); return true;
    case PLK_GATE_HADAMARD: L.u1(b[0], r, r, r, -r); return true;
    case PLK_GATE_S: inv ? Sd(b[0]) : S(b[0]); return true;
    case PLK_GATE_T: L.diag1(b[0], 1, cplx(std::cos(M_PI / 4), inv ? -std::sin(M_PI / 4) : std::sin(M_PI / 4))); return true;
    case PLK_GATE_PHASESHIFT: // exp(i t |1><1|): Jac = -2 Im <h|1><1|v>
        L.diag1(b[0], 1, expi(th));
        if (slot >= 0) L.grad_u1(slot, -sg, 0, 0, sg);
        return true;
    case PLK_GATE_RX:
        L.u1(b[0], c, -i1 * s, -i1 * s, c);
        if (slot >= 0) L.grad_u1(slot, 0, sg, 0, 0);
        return true;
    case PLK_GATE_RY:
        L.u1(b[0], c, -s, s, c);
        if (slot >= 0) L.grad_u1(slot, 0, 0, sg, 0);
        return true;
    case PLK_GATE_RZ:
        L.diag1(b[0], cplx(c, -s), cplx(c, s));
        if (slot >= 0) L.grad_u1(slot, 0, 0, 0, sg);
        return true;
    case PLK_GATE_ROT:
    case PLK_GATE_CROT: {
        if (op.num_params < 3 || !op.params) return false;
        const double phi = inv ? -op.params[2] : op.params[0], theta = inv ? -op.params[1] : op.params[1];
        const double omega = inv ? -op.params[0] : op.params[2];
        const double cc = std::cos(theta / 2), ss = std::sin(theta / 2);
        if (op.gate == PLK_GATE_ROT) {
            L.u1(b[0], expi(-(phi + omega) / 2) * cc, -expi((phi - omega) / 2) * ss, expi(-(phi - omega) / 2) * ss,
                 expi((phi + omega) / 2) * cc);
        } else { // table index bit 0: target, bit 1: control
            L.diag({b[1], b[0]}, {1, 1, expi(-phi / 2), expi(phi / 2)});
            L.cry(b[1], bit(b[0]), bit(b[0]), cc, ss);
            L.diag({b[1], b[0]}, {1, 1, expi(-omega / 2), expi(omega / 2)});
        }
        return true;
    }
    case PLK_GATE_CNOT: L.cx(b[0], b[1]); return true;
    case PLK_GATE_CY: Sd(b[1]); L.cx(b[0], b[1]); S(b[1]); return true;
    case PLK_GATE_CZ: L.diag({b[1], b[0]}, {1, 1, 1, -1}); return true;
    case PLK_GATE_SWAP: L.swap(b[0], b[1]); return true;
    case PLK_GATE_CONTROLLEDPHASESHIFT:
        L.diag({b[1], b[0]}, {1, 1, 1, expi(th)});
        if (slot >= 0) L.grad_diag(slot, -2 * sg, {0, 0, 0, 1});
        return true;
    case PLK_GATE_CRX:
        S(b[1]);
        L.cry(b[1], bit(b[0]), bit(b[0]), c, s);
        grad_cry(sg);
        Sd(b[1]);
        return true;
    case PLK_GATE_CRY:
        L.cry(b[1], bit(b[0]), bit(b[0]), c, s);
        grad_cry(sg);
        return true;
    case PLK_GATE_CRZ:
        L.diag({b[1], b[0]}, {1, 1, cplx(c, -s), cplx(c, s)});
        if (slot >= 0) L.grad_diag(slot, sg, {0, 0, 1, -1});
        return true;
    case PLK_GATE_ISINGXX:
    case PLK_GATE_ISINGYY: {
        const bool yy = op.gate == PLK_GATE_ISINGYY;
        if (yy) {
            Sd(b[0]);
            Sd(b[1]);
        }
        L.cx(b[0], b[1]);
        L.u1(b[0], c, -i1 * s, -i1 * s, c);
        if (slot >= 0) L.grad_u1(slot, 0, sg, 0, 0);
        L.cx(b[0], b[1]);
        if (yy) {
            S(b[0]);
            S(b[1]);
        }
        return true;
    }
    case PLK_GATE_ISINGXY: // the pair (01, 10) turns as RX(-t)
        L.cx(b[0], b[1]);
        S(b[0]);
        L.cry(b[0], bit(b[1]), bit(b[1]), c, -s);
        grad_cry(-sg);
        Sd(b[0]);
        L.cx(b[0], b[1]);
        return true;
    case PLK_GATE_ISINGZZ:
        L.diag({b[1], b[0]}, {cplx(c, -s), cplx(c, s), cplx(c, s), cplx(c, -s)});
        if (slot >= 0) L.grad_diag(slot, sg, {1, -1, -1, 1});
        return true;
    case PLK_GATE_SINGLEEXCITATION:
    case PLK_GATE_SINGLEEXCITATIONMINUS:
    case PLK_GATE_SINGLEEXCITATIONPLUS: {
        // after CX the pair (01, 10) is the target bit under b[1] = 1, and
        // 00, 11 have b[1] = 0
        L.cx(b[0], b[1]);
        L.cry(b[0], bit(b[1]), bit(b[1]), c, s);
        grad_cry(sg);
        if (op.gate != PLK_GATE_SINGLEEXCITATION) {
            const double k = op.gate == PLK_GATE_SINGLEEXCITATIONMINUS ? 1.0 : -1.0;
            L.diag1(b[1], cplx(c, -k * s), 1);
            if (slot >= 0) L.grad_u1(slot, 0.5 * k * sg, 0, 0, 0.5 * k * sg);
        }
        L.cx(b[0], b[1]);
        return true;
    }
    case PLK_GATE_DOUBLEEXCITATION:
    case PLK_GATE_DOUBLEEXCITATIONMINUS:
    case PLK_GATE_DOUBLEEXCITATIONPLUS: {
        // after the CXs the pair (0011, 1100) is the first bit under 011
        for (int j = 1; j < 4; j++) L.cx(b[0], b[j]);
        L.cry(b[0], bit(b[1]) | bit(b[2]) | bit(b[3]), bit(b[2]) | bit(b[3]), c, s);
        grad_cry(sg);
        if (op.gate != PLK_GATE_DOUBLEEXCITATION) {
            const double k = op.gate == PLK_GATE_DOUBLEEXCITATIONMINUS ? 1.0 : -1.0;
            const cplx e(c, -k * s);
            std::vector<double> g(8, 1.0);
            g[3] = 0; // table index: bit 0 b[3], bit 1 b[2], bit 2 b[1]
            L.diag({b[3], b[2], b[1]}, {e, e, e, 1, e, e, e, e});
            if (slot >= 0) L.grad_diag(slot, k * sg, g);
        }
        for (int j = 3; j >= 1; j--) L.cx(b[0], b[j]);
        return true;
    }
    case PLK_GATE_TOFFOLI: // X = RY(pi) Z under both controls
        L.diag({b[2], b[1], b[0]}, {1, 1, 1, 1, 1, 1, 1, -1});
        L.cry(b[2], bit(b[0]) | bit(b[1]), bit(b[0]) | bit(b[1]), 0, 1);
        return true;
    case PLK_GATE_CSWAP:
        L.cx(b[2], b[1]);
        L.diag({b[2], b[1], b[0]}, {1, 1, 1, 1, 1, 1, 1, -1});
        L.cry(b[2], bit(b[0]) | bit(b[1]), bit(b[0]) | bit(b[1]), 0, 1);
        L.cx(b[2], b[1]);
        return true;
    case PLK_GATE_MULTIRZ: {
        Prim p;
        p.kind = P_PAR;
        for (int j = 0; j < op.num_wires; j++) p.pmask |= 1u << (nq - 1 - (int)op.wires[j]);
        p.d[0] = cplx(c, -s);
        p.d[1] = cplx(c, s);
        if (slot >= 0) p.grads.push_back(Grad{slot, {0, 0, 0, sg}, {}, 1.0});
        L.v.push_back(p);
        return true;
    }
    default: return false;
    }
}

// primitives of the inverse, in application order
inline void invert(std::vector<Prim> &v) {
    std::reverse(v.begin(), v.end());
    for (Prim &p : v) {
        switch (p.kind) {
        case P_U1: {
            const cplx a = std::conj(p.m[0]), b = std::conj(p.m[2]), c = std::conj(p.m[1]), d = std::conj(p.m[3]);
            p.m[0] = a;
            p.m[1] = b;
            p.m[2] = c;
            p.m[3] = d;
            break;
        }
        case P_DIAG:
        case P_PAR:
            for (cplx &z : p.d) z = std::conj(z);
            break;
        case P_CRY: p.s = -p.s; break;
        default: break;
        }
    }
}

// -------------------------------------------------------------- scheduling --
// Access of a unit to a state bit: two units commute when every bit they share
// is accessed as D by both (block diagonal in it) or as F by both (flips).
enum Access : uint8_t { AC_N = 0, AC_D = 1, AC_F = 2 };

struct Term { // coef * (a sum) enters Jacobian slot
    int slot;
    double coef;
    int ref = -1;
};
struct ZTerm : Term { // the Walsh sum of the state bits in mask
    uint32_t mask;
    ZTerm(uint32_t m, int s, double c, int r = -1) : Term{s, c, r}, mask(m) {}
};

struct Unit {
    int kind = P_X; // P_* (P_U1: a run with a rotation; diagonal runs are P_DIAG)
    Prim p;
    cplx a0 = 1, a1 = 1, b0 = 1, b1 = 1; // U1: diag(b) RY(c, s) diag(a), |s| <= c
    bool has_a = false, has_b = false;
    // gradient terms (Jacobian slot, coefficient)
    std::vector<Term> gx, gy; // U1, CRY
    std::vector<ZTerm> gz;    // U1, DIAG, PAR
    int srun = -1, pool_a = -1, pool_b = -1; // symbolic: run, entries of a (diagonals: the entries) and b
    uint32_t bits = 0; // all state bits touched
    uint32_t need = 0; // bits that have to be in the tile
    uint32_t reg = 0;  // bits that have to be register bits
    int ngrad() const { return (gx.empty() ? 0 : 1) + (gy.empty() ? 0 : 1) + (int)gz.size(); }
};

struct Options {
    int T = 12;        // tile bits wanted (at most nq)
    int R = 4;         // register bits of a round
    int low = 3;       // lowest state bits in every tile (coalescing)
    int amp_bytes = 8; // bytes of an amplitude in shared memory (8: complex64, 16: double-float pairs)
    size_t max_blob = 20480;
};

class Compiler {
  public:
    Compiler(int nq, bool bwd, const Options &o, Symbols *sym = nullptr) : nq_(nq), bwd_(bwd), o_(o), sym_(sym) {
        T_ = std::min(o.T, nq);
        R_ = std::min(o.R, T_);
        last_.assign(nq, -1);
    }

    // primitives of one op, in application order of this sweep
    void add(const std::vector<Prim> &prims) {
        for (const Prim &p : prims) add_prim(p);
    }

    bool compile(TileProgram &P) {
        make_units();
        make_graph();
        P.nq = nq_;
        P.T = T_;
        P.R = R_;
        P.bwd = bwd_;
        P.nacc = 0;
        std::vector<int> ready;
        for (int i = 0; i < (int)units_.size(); i++)
            if (indeg_[i] == 0) ready.push_back(i);
        deg_.assign(units_.size(), 0);
        in_.assign(units_.size(), 0);
        used_.assign(groups_.size(), 0);
        pend_ = 1;
        last_table_ = Table{};
        size_t done = 0;
        std::vector<int> sel;
        std::vector<JacTerm> jac;
        while (done < units_.size()) {
            uint32_t bits = 0;
            select(ready, sel, bits);
            if (sel.empty()) return false;
            TilePass pass;
            int nacc = 0;
            const double pend = pend_;
            const Table last_table = last_table_;
            const size_t nf = sym_ ? sym_->factors.size() : 0, nt = sym_ ? sym_->tables.size() : 0;
            const size_t np = sym_ ? sym_->patches.size() : 0;
            for (;;) {
                jac.clear();
                if (sym_) {
                    sym_->factors.resize(nf);
                    sym_->tables.resize(nt);
                    sym_->patches.resize(np);
                }
                pend_ = pend;
                last_table_ = last_table;
                pass_ = (int)P.passes.size();
                jac0_ = P.jac.size();
                if (!build_pass(sel, bits, P.nacc, pass, jac, nacc)) return false;
                if (pass.blob.size() <= o_.max_blob || sel.size() <= 4) break;
                sel.resize(sel.size() * 3 / 4);
            }
            if (pass.blob.size() > o_.max_blob) return false;
            for (int i : sel) in_[i] = 1;
            ready.erase(std::remove_if(ready.begin(), ready.end(), [&](int i) { return in_[i] != 0; }), ready.end());
            for (int i : sel)
                for (int k = inc0_[i]; k < inc0_[i + 1]; k++) {
                    const Group &g = groups_[inc_[k].group];
                    if (--groups_[inc_[k].group].left > 0 || g.next < 0) continue;
                    for (int q = groups_[g.next].head; q >= 0; q = inc_[q].next)
                        if (--indeg_[inc_[q].unit] == 0 && !in_[inc_[q].unit]) insert_sorted(ready, inc_[q].unit);
                }
            for (int i : sel) in_[i] = 0;
            done += sel.size();
            P.nacc += nacc;
            P.jac.insert(P.jac.end(), jac.begin(), jac.end());
            P.passes.push_back(std::move(pass));
        }
        if (pend_ != 1) { // rotations after the last table: their factors go into it
            if (last_table_.pass < 0) return false;
            TilePass &p = P.passes[last_table_.pass];
            float *f = reinterpret_cast<float *>(
                p.blob.data() + reinterpret_cast<const TileHdr *>(p.blob.data())->off_tab + (size_t)last_table_.entry * 16);
            for (int k = 0; k < 4 << R_; k += 4)
                for (int q = 0; q < 2; q++) {
                    const double x = ((double)f[k + q] + (double)f[k + 2 + q]) * pend_;
                    f[k + q] = (float)x;
                    f[k + 2 + q] = (float)(x - (double)f[k + q]);
                }
            for (size_t i = last_table_.jac; i < P.jac.size(); i++) P.jac[i].coef /= pend_ * pend_;
        }
        return true;
    }

  private:
    int nq_, T_ = 0, R_ = 0;
    bool bwd_;
    Options o_;
    Symbols *sym_ = nullptr;
    std::vector<Prim> prims_;
    std::vector<int> last_; // last primitive touching each bit
    std::vector<Unit> units_;
    // The dependency graph.  The units on a state bit form groups that commute there
    // (all D, all F, or one unit); a unit waits, on each of its bits, for the whole group
    // before its own.  Groups, not pairs of units: lists of thousands of commuting
    // gates have as many groups as bits (whole calls on 20 qubits complex64, pairs /
    // groups: 10000 CZ 70 / 9.0 ms, 5000 CRZ and 5000 CNOT that share a wire 151 / 4.7).
    struct Group {
        Access a = AC_N;
        int prev = -1, next = -1; // groups of the same bit
        int left = 0;             // units not done
        int head = -1, tail = -1; // first and last incidence
    };
    struct Incidence { // a unit in a group
        int unit, group, next;
    };
    std::vector<Group> groups_;
    std::vector<Incidence> inc_;
    std::vector<int> inc0_;  // a unit's first incidence (and one past the last unit)
    std::vector<int> indeg_; // groups that a unit waits for
    std::vector<int> deg_;   // scratch: of these, inside a selection
    std::vector<int> used_;  // scratch: selected units of a group
    std::vector<char> in_;   // scratch: members of a selection
    // complex128: the state is pend_ times what the sweep holds
    double pend_ = 1;
    struct Table { // the last phase table: pass, first entry, Jacobian terms before it
        int pass = -1;
        uint32_t entry = 0;
        size_t jac = 0;
    } last_table_;
    int pass_ = 0;
    size_t jac0_ = 0;
    bool scaled() const { return o_.amp_bytes == 16; }

    static int popc(uint32_t x) { return __builtin_popcount(x); }
    static void insert_sorted(std::vector<int> &v, int x) { v.insert(std::lower_bound(v.begin(), v.end(), x), x); }

    static uint32_t bits_of(const Prim &p) {
        switch (p.kind) {
        case P_U1:
        case P_X: return 1u << p.t;
        case P_SWAP: return (1u << p.t) | (1u << p.t2);
        case P_CRY:
        case P_CX: return (1u << p.t) | p.cmask;
        case P_PAR: return p.pmask;
        default: {
            uint32_t m = 0;
            for (int i = 0; i < p.K; i++) m |= 1u << p.db[i];
            return m;
        }
        }
    }

    void add_prim(const Prim &p) {
        if (p.kind == P_U1) {
            const int l = last_[p.t];
            const int g = sym_ ? add_gate(p) : -1;
            if (l >= 0 && prims_[l].kind == P_U1) {
                if (sym_) {
                    sym_->gates[prims_[l].stail].next = g;
                    prims_[l].stail = g;
                    prims_[l].grads.insert(prims_[l].grads.end(), p.grads.begin(), p.grads.end());
                } else {
                    merge_u1(prims_[l], p);
                }
                return;
            }
            last_[p.t] = (int)prims_.size();
            prims_.push_back(p);
            prims_.back().shead = prims_.back().stail = g;
            return;
        }
        for (uint32_t m = bits_of(p); m; m &= m - 1) last_[__builtin_ctz(m)] = (int)prims_.size();
        prims_.push_back(p);
    }

    int add_gate(const Prim &p) {
        SymGate g;
        g.basis = p.sbasis;
        g.pidx = p.spidx;
        g.next = -1;
        // the form at the sample parameters of p is the form at all of them
        const bool diag = p.m[1] == 0.0 && p.m[2] == 0.0;
        const bool ry = !diag && p.m[0] == p.m[3] && p.m[1] == -p.m[2] && p.m[0].imag() == 0.0 && p.m[1].imag() == 0.0;
        g.form = diag ? GF_DIAG : ry ? GF_RY : GF_OTHER;
        for (int k = 0; k < 4; k++) {
            g.g[k] = p.grads.empty() ? 0.0 : p.grads[0].g[k];
            g.ref[k] = -1;
        }
        sym_->gates.push_back(g);
        return (int)sym_->gates.size() - 1;
    }

    // A run's type and the sums that its generators need, from the forms alone.
    void symbolic_run(Unit &u, Prim &p) {
        int first = -1, last = -1, n = 0, others = 0, diag_inside = 0;
        for (int g = p.shead; g >= 0; g = sym_->gates[g].next, n++)
            if (sym_->gates[g].form != GF_DIAG) {
                if (first < 0) first = n;
                last = n;
                others += sym_->gates[g].form == GF_OTHER;
            }
        n = 0;
        for (int g = p.shead; g >= 0; g = sym_->gates[g].next, n++)
            diag_inside += n > first && n < last && sym_->gates[g].form == GF_DIAG;
        SymRun r;
        r.head = p.shead;
        r.type = first < 0 ? RT_DIAG
                 : others || diag_inside || (first > 0 && last + 1 < n) ? RT_GENERAL
                 : last + 1 < n ? RT_LEFT
                                : RT_RIGHT;
        r.pool_a = r.pool_b = -1;
        if (r.type != RT_LEFT) {
            r.pool_a = sym_->npool;
            sym_->npool += 2;
        }
        if (r.type == RT_LEFT || r.type == RT_GENERAL) {
            r.pool_b = sym_->npool;
            sym_->npool += 2;
        }
        const uint32_t b = 1u << p.t;
        size_t grad = 0;
        int k = 0;
        for (int gi = p.shead; gi >= 0; gi = sym_->gates[gi].next, k++) {
            SymGate &g = sym_->gates[gi];
            if (g.g[0] == 0 && g.g[1] == 0 && g.g[2] == 0 && g.g[3] == 0) continue;
            const int slot = p.grads[grad++].slot;
            const bool start = first < 0 || k <= first; // only diagonals before it
            const bool plain = start && g.form == GF_DIAG;
            const bool only_y = g.form == GF_RY && r.type != RT_GENERAL;
            auto ref = [&](int c) { return g.ref[c] = sym_->nrefs++; };
            if (g.g[0] != 0) u.gz.push_back(ZTerm(0, slot, 1.0, ref(0)));
            if (!only_y) u.gz.push_back(ZTerm(b, slot, 1.0, ref(3)));
            if (!plain) {
                u.gy.push_back(Term{slot, 1.0, ref(2)});
                if (!only_y) u.gx.push_back(Term{slot, 1.0, ref(1)});
            }
        }
        u.srun = (int)sym_->runs.size();
        u.pool_a = r.pool_a;
        u.pool_b = r.pool_b;
        u.has_a = r.type == RT_RIGHT || r.type == RT_GENERAL;
        u.has_b = r.pool_b >= 0;
        if (r.type == RT_DIAG) {
            u.kind = p.kind = P_DIAG;
            p.K = 1;
            p.db[0] = p.t;
        }
        sym_->runs.push_back(r);
        u.p = std::move(p);
    }

    // a <- p a; p's generators (before p acts) in the frame of a's start
    static void merge_u1(Prim &a, const Prim &p) {
        for (Grad g : p.grads) {
            // W = V^dag (sum_k g_k sigma_k) V with V = a.m
            const cplx G[4] = {cplx(g.g[0] + g.g[3]), cplx(g.g[1], -g.g[2]), cplx(g.g[1], g.g[2]), cplx(g.g[0] - g.g[3])};
            cplx GV[4], W[4];
            for (int r = 0; r < 2; r++)
                for (int c = 0; c < 2; c++) GV[2 * r + c] = G[2 * r] * a.m[c] + G[2 * r + 1] * a.m[2 + c];
            for (int r = 0; r < 2; r++)
                for (int c = 0; c < 2; c++)
                    W[2 * r + c] = std::conj(a.m[r]) * GV[c] + std::conj(a.m[2 + r]) * GV[2 + c];
            g.g[0] = 0.5 * (W[0].real() + W[3].real());
            g.g[3] = 0.5 * (W[0].real() - W[3].real());
            g.g[1] = 0.5 * (W[1].real() + W[2].real());
            g.g[2] = 0.5 * (W[2].imag() - W[1].imag());
            a.grads.push_back(std::move(g));
        }
        cplx m[4];
        for (int r = 0; r < 2; r++)
            for (int c = 0; c < 2; c++) m[2 * r + c] = p.m[2 * r] * a.m[c] + p.m[2 * r + 1] * a.m[2 + c];
        std::copy(m, m + 4, a.m);
    }

    static bool near(cplx a, cplx b) { return std::fabs(a.real() - b.real()) < kTiny && std::fabs(a.imag() - b.imag()) < kTiny; }

    // m = g diag(b0, b1) [[c, -s], [s, c]] diag(a0, a1) with 0 < c, |s| <= c;
    // trivial sides where there are some
    static void split_u1(const cplx *m, Unit &u, cplx &g) {
        const double c = std::abs(m[0]), s0 = std::abs(m[2]);
        int best = -1;
        cplx best_g = 1;
        for (int k = 0; k < 2; k++) {
            const double s = k ? -s0 : s0;
            cplx a0 = 1, b0 = m[0] / c, b1 = m[2] / s, a1 = (m[3] / c) / b1, ph = 1;
            a1 /= std::abs(a1);
            b0 /= std::abs(b0);
            b1 /= std::abs(b1);
            if (near(b0, b1)) { // the common phase goes to the right, and out where that side is uniform too
                a0 = b0;
                a1 *= b0;
                b0 = b1 = 1;
            }
            if (near(a0, a1)) {
                if (near(b0, b1)) {
                    ph = a0;
                } else {
                    b0 *= a0;
                    b1 *= a0;
                }
                a0 = a1 = 1;
            }
            const bool ha = !(near(a0, 1) && near(a1, 1)), hb = !(near(b0, 1) && near(b1, 1));
            const int score = 2 - (ha ? 1 : 0) - (hb ? 1 : 0);
            if (score > best) {
                best = score;
                best_g = ph;
                u.p.c = c;
                u.p.s = s;
                u.a0 = a0;
                u.a1 = a1;
                u.b0 = b0;
                u.b1 = b1;
                u.has_a = ha;
                u.has_b = hb;
            }
        }
        g *= best_g;
    }

    static void add_gz(Unit &u, uint32_t mask, int slot, double coef) {
        if (std::fabs(coef) >= kTiny) u.gz.push_back(ZTerm(mask, slot, coef));
    }

    void make_units() {
        cplx g = 1; // phase of the whole state
        units_.reserve(prims_.size() + prims_.size() / 4 + 1);
        for (Prim &p : prims_) {
            Unit u;
            u.kind = p.kind;
            u.bits = bits_of(p);
            bool flip = false;
            if (sym_ && (p.kind == P_DIAG || p.kind == P_PAR || p.kind == P_CRY)) {
                const int n = p.kind == P_DIAG ? 1 << p.K : 2;
                u.pool_a = sym_->npool;
                sym_->npool += n;
                sym_->evals.push_back(SymEval{p.sbasis, p.spidx, n, u.pool_a});
            }
            if (p.kind == P_U1 && sym_) {
                symbolic_run(u, p);
            } else if (p.kind == P_U1) {
                const uint32_t b = 1u << p.t;
                if (std::norm(p.m[2]) > std::norm(p.m[0])) { // take an X out on the left
                    flip = true;
                    std::swap(p.m[0], p.m[2]);
                    std::swap(p.m[1], p.m[3]);
                }
                if (std::abs(p.m[1]) < kTiny && std::abs(p.m[2]) < kTiny) {
                    u.kind = p.kind = P_DIAG;
                    p.K = 1;
                    p.db[0] = p.t;
                    p.d[0] = p.m[0];
                    p.d[1] = p.m[3];
                    if (!flip) { // diagonal generators only
                        for (const Grad &e : p.grads) {
                            add_gz(u, 0, e.slot, e.g[0]);
                            add_gz(u, b, e.slot, e.g[3]);
                        }
                    }
                    bool off = false; // X or Y generators (a run that multiplies to a diagonal)
                    for (const Grad &e : p.grads) off = off || std::fabs(e.g[1]) >= kTiny || std::fabs(e.g[2]) >= kTiny;
                    if (off || flip) {
                        u.gz.clear();
                        if (!p.grads.empty()) { // measured on a rotation step by angle zero
                            u.kind = p.kind = P_U1;
                            u.p = p;
                            u.p.c = 1;
                            u.p.s = 0;
                            u.b0 = p.m[0];
                            u.b1 = p.m[3];
                            u.has_b = true;
                            add_u1_grads(u, p, b);
                        }
                    }
                    if (u.kind == P_DIAG && u.gz.empty() && near(p.d[0], p.d[1])) {
                        g *= p.d[0];
                        if (flip) push_x(p.t);
                        continue;
                    }
                    if (u.kind == P_DIAG) u.p = std::move(p);
                } else {
                    split_u1(p.m, u, g);
                    const double c = u.p.c, s = u.p.s;
                    u.p = p;
                    u.p.c = c;
                    u.p.s = s;
                    add_u1_grads(u, p, b);
                }
            } else {
                if (p.kind == P_CRY) {
                    for (const Grad &e : p.grads) u.gy.push_back(Term{e.slot, e.g[2]});
                } else if (p.kind == P_PAR) {
                    for (const Grad &e : p.grads) add_gz(u, p.pmask, e.slot, e.g[3]);
                } else if (p.kind == P_DIAG) {
                    for (const Grad &e : p.grads) // Walsh coefficients of the generator's diagonal
                        for (int w = 0; w < (1 << p.K); w++) {
                            double t = 0;
                            uint32_t mask = 0;
                            for (int i = 0; i < (1 << p.K); i++) t += (popc(i & w) & 1) ? -e.table[i] : e.table[i];
                            for (int i = 0; i < p.K; i++)
                                if (w >> i & 1) mask |= 1u << p.db[i];
                            add_gz(u, mask, e.slot, e.coef * t / (1 << p.K));
                        }
                }
                u.p = std::move(p);
            }
            const int t = u.p.t;
            push(std::move(u));
            if (flip) push_x(t);
        }
        prims_.clear();
        if (scaled()) { // some phase table has to take the rotations' factors
            bool turns = false, tables = false;
            for (const Unit &u : units_)
                if (u.kind == P_U1) {
                    turns = true;
                    tables = tables || u.has_a || u.has_b;
                }
            if (turns && !tables) {
                Unit u;
                u.kind = u.p.kind = P_DIAG;
                u.p.K = 1;
                u.p.d[0] = u.p.d[1] = 1;
                u.bits = 1;
                push(std::move(u));
            }
        }
        if (!near(g, 1)) { // into the first table there is
            for (Unit &u : units_) {
                if (u.kind == P_DIAG || u.kind == P_PAR) {
                    for (cplx &z : u.p.d) z *= g;
                } else if (u.kind == P_U1 && (u.has_a || u.has_b)) {
                    cplx &x = u.has_a ? u.a0 : u.b0, &y = u.has_a ? u.a1 : u.b1;
                    x *= g;
                    y *= g;
                } else {
                    continue;
                }
                return;
            }
            Unit u;
            u.kind = u.p.kind = P_DIAG;
            u.p.K = 1;
            u.p.d[0] = u.p.d[1] = g;
            u.bits = 1;
            push(std::move(u));
        }
    }

    // X and Y of the run's start as they stand after its right-hand phases:
    // X -> cos X + sin Y, Y -> cos Y - sin X
    static void add_u1_grads(Unit &u, const Prim &p, uint32_t b) {
        const cplx ph = u.a1 / u.a0;
        for (const Grad &e : p.grads) {
            const double gx = e.g[1] * ph.real() - e.g[2] * ph.imag();
            const double gy = e.g[1] * ph.imag() + e.g[2] * ph.real();
            if (std::fabs(gx) >= kTiny) u.gx.push_back(Term{e.slot, gx});
            if (std::fabs(gy) >= kTiny) u.gy.push_back(Term{e.slot, gy});
            add_gz(u, 0, e.slot, e.g[0]);
            add_gz(u, b, e.slot, e.g[3]);
        }
    }

    void push_x(int t) {
        Unit u;
        u.kind = u.p.kind = P_X;
        u.p.t = t;
        u.bits = 1u << t;
        push(std::move(u));
    }

    void push(Unit &&u) {
        switch (u.kind) {
        case P_U1:
        case P_CRY: u.need = u.reg = 1u << u.p.t; break;
        case P_CX:
        case P_X: u.need = 1u << u.p.t; break;
        case P_SWAP: u.need = u.bits; break;
        default: // diagonal: in registers where that is cheap to have
            if (popc(u.bits) <= R_ - 1) u.need = u.reg = u.bits;
            break;
        }
        units_.push_back(std::move(u));
    }

    static Access access(const Unit &u, int bit) {
        const uint32_t m = 1u << bit;
        switch (u.kind) {
        case P_DIAG:
        case P_PAR: return AC_D;
        case P_CRY: return (u.p.cmask & m) ? AC_D : AC_N;
        case P_CX: return (u.p.cmask & m) ? AC_D : AC_F;
        case P_X: return AC_F;
        default: return AC_N;
        }
    }

    void make_graph() {
        const int n = (int)units_.size();
        groups_.clear();
        inc_.clear();
        inc0_.assign(1, 0);
        indeg_.assign(n, 0);
        std::vector<int> last(nq_, -1); // present group of a bit
        for (int i = 0; i < n; i++) {
            for (uint32_t m = units_[i].bits; m; m &= m - 1) {
                const int b = __builtin_ctz(m), before = last[b];
                const Access a = access(units_[i], b);
                if (before < 0 || a == AC_N || groups_[before].a != a) {
                    Group g;
                    g.a = a;
                    g.prev = before;
                    last[b] = (int)groups_.size();
                    if (before >= 0) groups_[before].next = last[b];
                    groups_.push_back(g);
                }
                Group &g = groups_[last[b]];
                (g.tail < 0 ? g.head : inc_[g.tail].next) = (int)inc_.size();
                g.tail = (int)inc_.size();
                g.left++;
                if (g.prev >= 0) indeg_[i]++;
                inc_.push_back({i, last[b], -1});
            }
            inc0_.push_back((int)inc_.size());
        }
    }

    // the units of the next pass, in an order that respects the graph
    void select(const std::vector<int> &ready0, std::vector<int> &sel, uint32_t &bits) {
        std::vector<int> ready = ready0, touched, touched_groups;
        sel.clear();
        if (T_ >= nq_) bits = nq_ >= 32 ? 0xffffffffu : (1u << nq_) - 1;
        else bits = (1u << o_.low) - 1;
        int acc = 0;
        size_t from = 0; // those before it do not fit, and will not while `bits` stays as it is
        while (!ready.empty() && (int)sel.size() < kMaxUnits) {
            int pick = -1;
            for (int pass = 0; pass < 2 && pick < 0; pass++)
                for (size_t r = pass == 0 ? from : 0; r < ready.size() && pick < 0; r++) {
                    const Unit &u = units_[ready[r]];
                    if (acc + u.ngrad() > kMaxAcc) continue;
                    if (pass == 0 ? (u.need & ~bits) == 0 : popc(bits | u.need) <= T_) pick = (int)r;
                }
            if (pick < 0) break;
            const int i = ready[pick];
            ready.erase(ready.begin() + pick);
            from = (units_[i].need & ~bits) ? 0 : (size_t)pick;
            bits |= units_[i].need;
            acc += units_[i].ngrad();
            sel.push_back(i);
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) {
                const int gi = inc_[k].group;
                const Group &g = groups_[gi];
                if (used_[gi]++ == 0) touched_groups.push_back(gi);
                if (used_[gi] < g.left || g.next < 0) continue;
                for (int q = groups_[g.next].head; q >= 0; q = inc_[q].next) {
                    const int s = inc_[q].unit;
                    if (deg_[s]++ == 0) touched.push_back(s);
                    if (deg_[s] < indeg_[s]) continue;
                    const auto at = std::lower_bound(ready.begin(), ready.end(), s);
                    from = std::min(from, (size_t)(at - ready.begin()));
                    ready.insert(at, s);
                }
            }
        }
        for (int s : touched) deg_[s] = 0;
        for (int g : touched_groups) used_[g] = 0;
        for (int b = 0; b < nq_ && popc(bits) < T_; b++) bits |= 1u << b; // fill with low bits
    }

    // -------------------------------------------------------------- passes --
    using Terms = std::vector<Term>;

    struct Factor { // a diagonal factor of a table: a unit's, or one side of a run
        const Unit *u = nullptr;
        int bit = 0;
        cplx e0 = 1, e1 = 1;
        int pool = -1;
    };
    enum StepKind { SK_RY, SK_CRY, SK_TAB, SK_INDEX };
    struct Step {
        int kind = SK_RY;
        const Unit *u = nullptr; // RY, CRY, INDEX
        uint32_t support = 0;    // TAB, INDEX: state bits
        std::vector<Factor> f;   // TAB
        std::vector<ZTerm> gz;   // TAB
    };

    // A diagonal factor joins a table that it commutes to (the earliest, or for
    // the left side of a run the latest), else opens one.
    static Step &table_for(std::vector<Step> &st, uint32_t m, bool latest) {
        Step *t = nullptr;
        for (size_t i = st.size(); i-- > 0 && !(t && latest);) {
            if (st[i].kind == SK_TAB) t = &st[i];
            else if (st[i].kind != SK_INDEX && (m >> st[i].u->p.t & 1)) break;
        }
        if (!t) {
            st.emplace_back();
            t = &st.back();
            t->kind = SK_TAB;
        }
        t->support |= m;
        return *t;
    }

    // A rotation goes before trailing tables that leave its bit alone, so that
    // later phases on that bit still find them.
    static void place_turn(std::vector<Step> &st, const Unit &u) {
        size_t p = st.size();
        while (p > 0 && st[p - 1].kind >= SK_TAB && !(st[p - 1].support >> u.p.t & 1)) p--;
        Step r;
        r.kind = u.kind == P_U1 ? SK_RY : SK_CRY;
        r.u = &u;
        st.insert(st.begin() + p, std::move(r));
    }

    void place(std::vector<Step> &st, const Unit &u, uint32_t regs) const {
        if (u.kind == P_U1 || u.kind == P_CRY) {
            const uint32_t b = 1u << u.p.t;
            if (u.has_a || !u.gz.empty()) {
                Step &t = table_for(st, b, false);
                if (u.has_a) t.f.push_back(Factor{nullptr, u.p.t, u.a0, u.a1, u.pool_a});
                t.gz.insert(t.gz.end(), u.gz.begin(), u.gz.end());
            }
            place_turn(st, u);
            if (u.has_b) table_for(st, b, true).f.push_back(Factor{nullptr, u.p.t, u.b0, u.b1, u.pool_b});
        } else if ((u.bits & ~regs) == 0) {
            Step &t = table_for(st, u.bits, false);
            t.f.push_back(Factor{&u, 0, 1, 1, u.pool_a});
            t.gz.insert(t.gz.end(), u.gz.begin(), u.gz.end());
        } else {
            Step d;
            d.kind = SK_INDEX;
            d.u = &u;
            d.support = u.bits;
            st.push_back(std::move(d));
        }
    }

    uint32_t swizzle(uint32_t p) const {
        if (o_.amp_bytes == 8) return p ^ ((p >> 4 ^ p >> 8 ^ p >> 12) & 15u);
        return p ^ ((p >> 3 ^ p >> 6 ^ p >> 9 ^ p >> 12) & 7u);
    }

    static bool is_perm(const Unit &u) { return u.kind == P_CX || u.kind == P_X || u.kind == P_SWAP; }

    // pass under construction
    struct Out {
        std::vector<int> tbits;      // state bit of tile bit k
        std::vector<int> pos;        // tile bit of a state bit, -1 outside
        std::vector<uint32_t> col;   // map: tile index x -> slot A x + xc, columns of A
        uint32_t xc = 0;
        std::vector<uint32_t> out;   // x of the last round -> x now: columns, constant
        uint32_t outc = 0;
        std::vector<uint32_t> out_ev; // its constant's event masks, from event out_ev0 on
        size_t ev0 = 0;              // events before this one belong to earlier rounds
        std::vector<int> last_tb, last_rb; // thread and register bits of the last round
        std::vector<TileRound> rounds;
        std::vector<TileStage> stages;
        std::vector<TileEvent> events;
        std::vector<TileIndex> index;
        std::vector<float> tab;
    };

    uint32_t tab_pos(const Out &o) const { return (uint32_t)(o.tab.size() * sizeof(float) / o_.amp_bytes); }
    void put(Out &o, cplx z) const {
        const float rh = (float)z.real(), ih = (float)z.imag();
        o.tab.push_back(rh);
        o.tab.push_back(ih);
        if (o_.amp_bytes == 16) {
            o.tab.push_back((float)(z.real() - (double)rh));
            o.tab.push_back((float)(z.imag() - (double)ih));
        }
    }
    static void put2(float *f, double x) {
        f[0] = (float)x;
        f[1] = (float)(x - (double)f[0]);
    }

    // entries combined by exclusive or, each from the one without its lowest bit
    template <class T, class F> static void span(T *lo, T *hi, int n, F column) {
        for (int l = 0; l < 32; l++) {
            const int r = l & (l - 1), k = l ? __builtin_ctz(l) : 0;
            lo[l] = l ? (T)(lo[r] ^ (k < n ? column(k) : 0)) : (T)0;
        }
        for (int h = 0; h < 16; h++) {
            const int r = h & (h - 1), k = 5 + (h ? __builtin_ctz(h) : 0);
            hi[h] = h ? (T)(hi[r] ^ (k < n ? column(k) : 0)) : (T)0;
        }
    }

    uint32_t deposit(const Out &o, uint32_t x) const {
        uint32_t g = 0;
        for (; x; x &= x - 1) g |= 1u << o.tbits[__builtin_ctz(x)];
        return g;
    }

    // state index of (thread, register) through the columns c
    uint32_t add_index(Out &o, const std::vector<int> &tb, const std::vector<int> &rb, const std::vector<uint32_t> &c,
                       uint32_t constant) const {
        TileIndex x;
        std::memset(&x, 0, sizeof(x));
        span(x.lo, x.hi, (int)tb.size(), [&](int k) { return deposit(o, c[tb[k]]); });
        for (int i = 0; i < R_; i++) x.r[i] = deposit(o, c[rb[i]]);
        x.c = deposit(o, constant);
        o.index.push_back(x);
        return (uint32_t)o.index.size() - 1;
    }

    // do the lanes cover the lowest state bits?
    bool coalesced(const std::vector<int> &tb) const {
        const int n = std::min(o_.low, (int)tb.size());
        for (int k = 0; k < n; k++)
            if (std::find(tb.begin(), tb.begin() + std::min<size_t>(5, tb.size()), k) ==
                tb.begin() + std::min<size_t>(5, tb.size()))
                return false;
        return true;
    }

    static void identity(std::vector<uint32_t> &c, int n) {
        c.resize(n);
        for (int k = 0; k < n; k++) c[k] = 1u << k;
    }

    // A round on the register bits `regs` with the present map.
    TileRound &open_round(Out &o, uint32_t regs, bool low_lanes) const {
        TileRound r;
        std::memset(&r, 0, sizeof(r));
        std::vector<int> rest, &tb = o.last_tb, &rb = o.last_rb;
        tb.clear();
        rb.clear();
        for (int k = 0; k < T_; k++) (regs >> o.tbits[k] & 1 ? rb : rest).push_back(k);
        // lanes first get bits whose columns are independent in the bank bits,
        // so that the amplitudes of a memory wavefront lie in different banks
        if (low_lanes) {
            tb = rest;
        } else {
            const uint32_t bank = o_.amp_bytes == 8 ? 15u : 7u;
            std::vector<int> later;
            uint32_t basis[4];
            int nb = 0;
            for (int k : rest) {
                uint32_t v = swizzle(o.col[k]) & bank;
                for (int i = 0; i < nb; i++) v = std::min(v, v ^ basis[i]);
                if (v) {
                    basis[nb++] = v;
                    tb.push_back(k);
                } else {
                    later.push_back(k);
                }
            }
            tb.insert(tb.end(), later.begin(), later.end());
        }
        const uint32_t ab = (uint32_t)o_.amp_bytes;
        span(r.lo, r.hi, (int)tb.size(), [&](int k) { return swizzle(o.col[tb[k]]) * ab; });
        for (int i = 0; i < R_; i++) r.rcol[i] = (uint16_t)(swizzle(o.col[rb[i]]) * ab);
        r.xorc = (uint16_t)(swizzle(o.xc) * ab);
        r.ev0 = (uint16_t)o.ev0;
        r.nev = (uint16_t)(o.events.size() - o.ev0);
        o.ev0 = o.events.size();
        r.stage0 = (uint16_t)o.stages.size();
        r.idx = 0xffff;
        identity(o.out, T_);
        o.outc = 0;
        o.out_ev.clear();
        o.rounds.push_back(r);
        return o.rounds.back();
    }

    uint32_t top_bits(const Out &o) const {
        uint32_t m = 0;
        for (int i = 0; i < R_; i++) m |= 1u << o.tbits[T_ - 1 - i];
        return m;
    }

    bool emit_round(Out &o, const std::vector<Step> &st, uint32_t regs, int acc0, std::vector<JacTerm> &jac,
                    int &nacc) {
        if (o.rounds.empty()) { // reads the state
            const uint32_t c = o.xc;
            std::vector<uint32_t> col = o.col;
            open_round(o, regs, false);
            if (!coalesced(o.last_tb)) { // through a round of its own
                o.rounds.clear();
                o.ev0 = 0;
                open_round(o, top_bits(o), true);
                add_index(o, o.last_tb, o.last_rb, col, c);
                open_round(o, regs, false);
            } else {
                add_index(o, o.last_tb, o.last_rb, col, c);
            }
        } else {
            open_round(o, regs, false);
        }
        TileRound &r = o.rounds.back();
        int rstate[kMaxRegBits];
        for (int i = 0; i < R_; i++) rstate[i] = o.tbits[o.last_rb[i]];
        const int amps = 1 << R_;
        bool want_index = false;
        auto acc = [&](const Terms &t) -> int16_t {
            if (t.empty()) return -1;
            for (const Term &e : t) jac.push_back(JacTerm{e.slot, acc0 + nacc, e.coef * pend_ * pend_, e.ref});
            return (int16_t)nacc++;
        };
        auto reg_of = [&](int state_bit) {
            for (int i = 0; i < R_; i++)
                if (rstate[i] == state_bit) return i;
            return -1;
        };
        auto reg_mask = [&](uint32_t m) {
            uint32_t q = 0;
            for (int i = 0; i < R_; i++) q |= (m >> rstate[i] & 1) << i;
            return q;
        };
        TileStage cur;
        const Unit *turn[4]; // rotations of the stage by bit
        bool any = false;
        auto reset = [&]() {
            std::memset(&cur, 0, sizeof(cur));
            for (int i = 0; i < 4; i++) {
                cur.acc_y[i] = cur.acc_x[i] = cur.acc_zb[i] = -1;
                turn[i] = nullptr;
            }
            cur.acc_z = cur.sacc = -1;
            any = false;
        };
        // rotations run by ascending bit, each measured before it runs
        auto turns = [&]() {
            for (int b = 0; b < R_; b++) {
                if (!turn[b]) continue;
                const Unit &u = *turn[b];
                cur.ry |= (uint8_t)(1u << b);
                if (sym_)
                    sym_->patches.push_back(SymPatch{
                        pass_, (uint32_t)(o.stages.size() * sizeof(TileStage) + offsetof(TileStage, rot) + 16 * b), 0,
                        u.srun, 0});
                if (scaled()) {
                    put2(cur.rot[b], u.p.s / u.p.c);
                } else {
                    put2(cur.rot[b], u.p.s / (1.0 + u.p.c));
                    put2(cur.rot[b] + 2, u.p.s);
                }
                cur.acc_y[b] = acc(u.gy);
                cur.acc_x[b] = acc(u.gx);
                cur.sums |= (uint8_t)((cur.acc_y[b] >= 0 ? 1 : 0) | (cur.acc_x[b] >= 0 ? 2 : 0));
                if (scaled()) pend_ *= u.p.c;
                turn[b] = nullptr;
            }
        };
        auto flush = [&]() {
            turns();
            if (any) o.stages.push_back(cur);
            reset();
        };
        // A stage that begins without a table gets one when the sweep holds more
        // than 2^8 times the state.  A stage turns at most kMaxRegBits bits by at
        // most sqrt(2) each, so what is held stays within 2^10, and a sum's
        // products within 2^20: controlled rotations between rotations, which meet
        // no phase, reached 2^64 and 2^128 when this was looked at once per round.
        auto begin = [&]() {
            if (!any && pend_ < 1.0 / 256) {
                cur.table |= 2;
                cur.tab = (uint16_t)tab_pos(o);
                for (int j = 0; j < amps; j++) put(o, pend_);
                pend_ = 1;
                last_table_ = Table{pass_, cur.tab, jac0_ + jac.size()};
            }
            any = true;
        };
        reset();
        std::vector<std::pair<uint32_t, const ZTerm *>> z;
        for (const Step &s : st) {
            if (s.kind == SK_TAB) {
                if (any) flush();
                any = true;
                const double scale = pend_;
                if (!s.f.empty() || pend_ < 1.0 / 256) {
                    cur.table |= 2;
                    cur.tab = (uint16_t)tab_pos(o);
                    cplx e[kMaxAmps];
                    for (int j = 0; j < amps; j++) e[j] = pend_;
                    pend_ = 1;
                    if (sym_) {
                        sym_->tables.push_back(SymTable{pass_, (uint32_t)(cur.tab * o_.amp_bytes),
                                                        (int32_t)sym_->factors.size(), (int32_t)s.f.size()});
                        for (const Factor &f : s.f) {
                            SymFactor q;
                            std::memset(&q, 0, sizeof(q));
                            q.pool = f.pool;
                            if (!f.u) {
                                q.K = 1;
                                q.reg[0] = (uint8_t)reg_of(f.bit);
                            } else if (f.u->kind == P_PAR) {
                                q.K = -1;
                                q.mask = (uint8_t)reg_mask(f.u->p.pmask);
                            } else {
                                q.K = (int8_t)f.u->p.K;
                                for (int i = 0; i < f.u->p.K; i++) q.reg[i] = (uint8_t)reg_of(f.u->p.db[i]);
                            }
                            sym_->factors.push_back(q);
                        }
                    }
                    for (const Factor &f : s.f) {
                        if (!f.u) {
                            const int i = reg_of(f.bit);
                            for (int j = 0; j < amps; j++) e[j] *= (j >> i & 1) ? f.e1 : f.e0;
                        } else if (f.u->kind == P_PAR) {
                            const uint32_t m = reg_mask(f.u->p.pmask);
                            for (int j = 0; j < amps; j++) e[j] *= f.u->p.d[popc(j & m) & 1];
                        } else {
                            int rg[3] = {0, 0, 0};
                            for (int q = 0; q < f.u->p.K; q++) rg[q] = reg_of(f.u->p.db[q]);
                            for (int j = 0; j < amps; j++) {
                                int li = 0;
                                for (int q = 0; q < f.u->p.K; q++) li |= (j >> rg[q] & 1) << q;
                                e[j] *= f.u->p.d[li];
                            }
                        }
                    }
                    for (int j = 0; j < amps; j++) put(o, e[j]);
                }
                if (!s.gz.empty()) { // accumulators by ascending register mask
                    cur.table |= 1;
                    z.clear();
                    for (const ZTerm &e : s.gz) z.push_back({reg_mask(e.mask), &e});
                    std::stable_sort(z.begin(), z.end(), [](const auto &x, const auto &y) { return x.first < y.first; });
                    for (size_t i = 0; i < z.size(); i++) {
                        if (i == 0 || z[i].first != z[i - 1].first) {
                            if (cur.acc_z < 0) cur.acc_z = (int16_t)nacc;
                            cur.zsel |= (uint16_t)(1u << z[i].first);
                            nacc++;
                        }
                        jac.push_back(JacTerm{z[i].second->slot, acc0 + nacc - 1, z[i].second->coef * scale * scale, z[i].second->ref});
                    }
                    if ((cur.zsel & ~0x0116u) == 0) { // masks 1, 2, 4, 8
                        int next = cur.acc_z;
                        for (int b = 0; b < 4; b++)
                            if (cur.zsel >> (1 << b) & 1) cur.acc_zb[b] = (int16_t)next++;
                    }
                }
                if (cur.table & 2) last_table_ = Table{pass_, cur.tab, jac0_ + jac.size()};
            } else if (s.kind == SK_RY) {
                const int b = reg_of(s.u->p.t);
                if (cur.special || turn[b]) flush();
                begin();
                turn[b] = s.u;
            } else {
                if (cur.special) flush();
                turns();
                begin();
                const Unit &u = *s.u;
                if (s.kind == SK_CRY) {
                    cur.special = TS_CRY;
                    cur.bit = (uint8_t)reg_of(u.p.t);
                    const uint32_t cm = reg_mask(u.p.cmask), cv = reg_mask(u.p.cval);
                    for (int j = 0; j < amps; j++)
                        if ((j & cm) == cv) cur.jact |= (uint16_t)(1u << j);
                    cur.cmask = u.p.cmask & ~regs;
                    cur.cval = u.p.cval & ~regs;
                    want_index = want_index || cur.cmask != 0;
                    if (sym_)
                        sym_->patches.push_back(SymPatch{
                            pass_, (uint32_t)(o.stages.size() * sizeof(TileStage) + offsetof(TileStage, coef)), 1, u.pool_a,
                            2});
                    put2(cur.coef, u.p.c);
                    put2(cur.coef + 2, u.p.s);
                    cur.sacc = acc(u.gy);
                } else {
                    want_index = true;
                    cur.stab = (uint16_t)tab_pos(o);
                    if (sym_)
                        sym_->patches.push_back(SymPatch{pass_, (uint32_t)(cur.stab * o_.amp_bytes), 2, u.pool_a,
                                                         u.kind == P_PAR ? 2 : 1 << u.p.K});
                    if (u.kind == P_PAR) {
                        cur.special = TS_PAR;
                        cur.cmask = u.p.pmask;
                        put(o, u.p.d[0]);
                        put(o, u.p.d[1]);
                        Terms g;
                        for (const ZTerm &e : u.gz) g.push_back(Term{e.slot, e.coef, e.ref});
                        cur.sacc = acc(g);
                    } else {
                        cur.special = TS_DIAG;
                        cur.K = (uint8_t)u.p.K;
                        for (int q = 0; q < u.p.K; q++) cur.cmask |= (uint32_t)u.p.db[q] << (5 * q);
                        for (int q = 0; q < (1 << u.p.K); q++) put(o, u.p.d[q]);
                        if (u.p.grads.size() > 1) return false;
                        for (const Grad &e : u.p.grads) {
                            cur.gtab = (uint32_t)o.tab.size();
                            for (double x : e.table) o.tab.push_back((float)x);
                            cur.sacc = acc(Terms{Term{e.slot, e.coef}});
                        }
                        while (o.tab.size() % 4) o.tab.push_back(0.0f); // tables are read 16 bytes at a time
                    }
                }
            }
        }
        flush();
        r.nstages = (uint16_t)(o.stages.size() - r.stage0);
        if (want_index) {
            std::vector<uint32_t> id;
            identity(id, T_);
            const std::vector<int> tb = o.last_tb, rb = o.last_rb;
            o.rounds.back().idx = (uint16_t)add_index(o, tb, rb, id, 0);
        }
        return true;
    }

    // composes an index map into the tile's map (and into the map from the
    // last round's indices to the present ones)
    void compose(Out &o, const Unit &u) const {
        const int t = o.pos[u.p.t];
        auto on_out = [&](auto f) {
            for (uint32_t &x : o.out) x = f(x);
            for (uint32_t &x : o.out_ev) x = f(x);
            o.outc = f(o.outc);
        };
        if (u.kind == P_X) {
            o.xc ^= o.col[t];
            o.outc ^= 1u << t;
        } else if (u.kind == P_SWAP) {
            const int q = o.pos[u.p.t2];
            std::swap(o.col[t], o.col[q]);
            on_out([&](uint32_t x) {
                const uint32_t d = (x >> t ^ x >> q) & 1u;
                return x ^ (d << t) ^ (d << q);
            });
        } else {
            const int cb = __builtin_ctz(u.p.cmask), c = o.pos[cb];
            if (c >= 0) {
                o.col[c] ^= o.col[t];
                on_out([&](uint32_t x) { return x ^ ((x >> c & 1u) << t); });
            } else {
                o.events.push_back(TileEvent{(uint16_t)(swizzle(o.col[t]) * o_.amp_bytes), (uint16_t)cb,
                                             deposit(o, o.col[t])});
                o.out_ev.push_back(1u << t);
            }
        }
    }

    bool build_pass(const std::vector<int> &sel, uint32_t bits, int acc0, TilePass &pass, std::vector<JacTerm> &jac,
                    int &nacc) {
        Out o;
        o.pos.assign(32, -1);
        for (int b = 0; b < nq_; b++)
            if (bits >> b & 1) {
                o.pos[b] = (int)o.tbits.size();
                o.tbits.push_back(b);
            }
        if ((int)o.tbits.size() != T_) return false;
        identity(o.col, T_);
        identity(o.out, T_);
        nacc = 0;
        for (int i : sel) {
            in_[i] = 1;
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) used_[inc_[k].group]++;
        }
        std::vector<int> ready;
        for (int i : sel) {
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) {
                const int before = groups_[inc_[k].group].prev;
                deg_[i] += before >= 0 && used_[before] > 0;
            }
            if (deg_[i] == 0) insert_sorted(ready, i);
        }
        size_t left = sel.size();
        // a group's selected units that are left, counted down from its units not done:
        // the next group is in the selection only where all of them are
        for (int i : sel)
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) used_[inc_[k].group] = groups_[inc_[k].group].left;
        auto finish = [&](size_t r) {
            const int i = ready[r];
            ready.erase(ready.begin() + r);
            left--;
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) {
                const int gi = inc_[k].group, after = groups_[gi].next;
                if (--used_[gi] > 0 || after < 0) continue;
                for (int q = groups_[after].head; q >= 0; q = inc_[q].next)
                    if (in_[inc_[q].unit] && --deg_[inc_[q].unit] == 0) insert_sorted(ready, inc_[q].unit);
            }
        };
        bool ok = true;
        std::vector<Step> st;
        while (left > 0 && ok) {
            for (size_t r = 0; r < ready.size();) { // index maps: composed, nothing moves
                if (is_perm(units_[ready[r]])) {
                    compose(o, units_[ready[r]]);
                    finish(r);
                    r = 0;
                } else {
                    r++;
                }
            }
            if (left == 0) break;
            st.clear();
            uint32_t regs = 0;
            for (;;) {
                int pick = -1;
                for (int p = 0; p < 2 && pick < 0; p++)
                    for (size_t r = 0; r < ready.size() && pick < 0; r++) {
                        const Unit &u = units_[ready[r]];
                        if (is_perm(u)) continue;
                        if (p == 0 ? (u.reg & ~regs) == 0 : popc(regs | u.reg) <= R_) pick = (int)r;
                    }
                if (pick < 0) break;
                const Unit &u = units_[ready[pick]];
                regs |= u.reg;
                finish(pick);
                place(st, u, regs);
            }
            for (int k = T_ - 1; k >= 0 && popc(regs) < R_; k--) regs |= 1u << o.tbits[k];
            ok = !st.empty() && emit_round(o, st, regs, acc0, jac, nacc);
        }
        for (int i : sel) {
            in_[i] = 0;
            deg_[i] = 0;
            for (int k = inc0_[i]; k < inc0_[i + 1]; k++) used_[inc_[k].group] = 0;
        }
        if (!ok || nacc > kMaxAcc * 2) return false;
        // the last round writes the state: through the map from its indices to
        // the present ones, or, where its lanes do not cover the lowest state
        // bits, in a round of its own
        TileHdr h;
        std::memset(&h, 0, sizeof(h));
        if (o.rounds.empty()) { // index maps only
            open_round(o, top_bits(o), true);
            add_index(o, o.last_tb, o.last_rb, o.col, o.xc);
        } else if (!coalesced(o.last_tb)) {
            open_round(o, top_bits(o), true);
        }
        h.ev_store0 = (int32_t)o.ev0;
        h.nev = (int32_t)o.events.size();
        for (size_t k = 0; k < o.out_ev.size(); k++) o.events[o.ev0 + k].gmask = deposit(o, o.out_ev[k]);
        h.load_idx = 0;
        {
            const std::vector<int> tb = o.last_tb, rb = o.last_rb;
            h.store_idx = add_index(o, tb, rb, o.out, o.outc);
        }
        h.T = T_;
        h.R = R_;
        h.nq = nq_;
        h.nrounds = (int32_t)o.rounds.size();
        h.nstages = (int32_t)o.stages.size();
        h.nacc = nacc;
        h.acc0 = acc0;
        for (int k = 0; k < T_; k++) h.gpos[k] = (uint8_t)o.tbits[k];
        size_t at = sizeof(TileHdr);
        auto area = [&](size_t bytes) {
            const size_t p = at;
            at += (bytes + 15) & ~(size_t)15;
            return (uint32_t)p;
        };
        h.off_rounds = area(o.rounds.size() * sizeof(TileRound));
        h.off_stages = area(o.stages.size() * sizeof(TileStage));
        h.off_events = area(o.events.size() * sizeof(TileEvent));
        h.off_index = area(o.index.size() * sizeof(TileIndex));
        h.off_tab = area(o.tab.size() * sizeof(float));
        h.bytes = (uint32_t)at;
        if (sym_) { // offsets within the blob
            for (size_t i = sym_->tables.size(); i-- > 0 && sym_->tables[i].pass == pass_;) sym_->tables[i].off += h.off_tab;
            for (size_t i = sym_->patches.size(); i-- > 0 && sym_->patches[i].pass == pass_;)
                sym_->patches[i].off += sym_->patches[i].kind == 2 ? h.off_tab : h.off_stages;
        }
        pass.blob.assign(at, 0);
        auto cp = [&](uint32_t off, const void *src, size_t bytes) {
            if (bytes) std::memcpy(pass.blob.data() + off, src, bytes);
        };
        cp(0, &h, sizeof(h));
        cp(h.off_rounds, o.rounds.data(), o.rounds.size() * sizeof(TileRound));
        cp(h.off_stages, o.stages.data(), o.stages.size() * sizeof(TileStage));
        cp(h.off_events, o.events.data(), o.events.size() * sizeof(TileEvent));
        cp(h.off_index, o.index.data(), o.index.size() * sizeof(TileIndex));
        cp(h.off_tab, o.tab.data(), o.tab.size() * sizeof(float));
        return true;
    }
};

} // namespace tile
} // namespace plk
