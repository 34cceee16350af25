// The rule for adjoint sweeps of several observables (csrc/sweep_cost.hpp) on the
// programs that the compiler makes, for tests/test_sweep_cost_cpu.py.
#include "sweep_cost.hpp"

using namespace plk::tile;

// 1: tiles, 0: op by op, -1: not compiled
extern "C" int tiles_chosen(int nq, int c64, int nobs, const plk_op *ops, int nops) {
    Options o;
    o.T = 11;
    o.R = c64 ? 4 : 3;
    o.low = c64 ? 3 : 2;
    o.amp_bytes = c64 ? 8 : 16;
    Compiler c(nq, true, o);
    std::vector<SweptOp> swept;
    int slot = 0;
    for (int i = 0; i < nops; i++) slot += ops[i].num_params > 0;
    for (int i = nops - 1; i >= 0; i--) {
        Lowered L;
        const bool t = ops[i].num_params > 0;
        if (!lower_op(ops[i], nq, t ? --slot : -1, L)) return -1;
        invert(L.v);
        c.add(L.v);
        swept.push_back({ops[i].gate, t});
    }
    TileProgram P;
    if (!c.compile(P)) return -1;
    return tiles_pay(nobs, c64 != 0, P, swept);
}
