// How far the numbers that a complex128 sweep holds may stand above the state:
// its rotations are [[1, -t], [t, 1]], each sqrt(1 + t^2) too large, until a
// phase table takes the factors back.  Built by tests/test_tile_growth_cpu.py.
#include <cmath>
#include <cstring>

#include "tile_program.hpp"

using namespace plk::tile;

// The largest factor within the program, rounded up to what all of a stage's
// rotations give, as log2; `left` is the factor at its end.  Negative: not compiled.
extern "C" double tile_growth(int nq, int T, int R, int low, int bwd, const plk_op *ops, int nops, const int64_t *slot,
                              double *left) {
    Options o;
    o.T = T;
    o.R = R;
    o.low = low;
    o.amp_bytes = 16;
    Compiler c(nq, bwd != 0, o);
    for (int k = 0; k < nops; k++) {
        const int i = bwd ? nops - 1 - k : k;
        Lowered L;
        if (!lower_op(ops[i], nq, bwd ? (int)slot[i] : -1, L)) return -1;
        if (bwd) invert(L.v);
        c.add(L.v);
    }
    TileProgram P;
    if (!c.compile(P)) return -1;
    double now = 0, most = 0;
    for (const TilePass &ps : P.passes) {
        const unsigned char *b = ps.blob.data();
        const TileHdr &h = *reinterpret_cast<const TileHdr *>(b);
        const TileStage *S = reinterpret_cast<const TileStage *>(b + h.off_stages);
        const TileRound *rounds = reinterpret_cast<const TileRound *>(b + h.off_rounds);
        for (int r = 0; r < h.nrounds; r++)
            for (int k = 0; k < rounds[r].nstages; k++) {
                const TileStage &st = S[rounds[r].stage0 + k];
                if (st.table & 2) {
                    float e[4];
                    std::memcpy(e, b + h.off_tab + (size_t)st.tab * 16, sizeof(e));
                    now += std::log2(std::hypot((double)e[0] + e[2], (double)e[1] + e[3]));
                    most = std::max(most, now);
                }
                for (int i = 0; i < h.R; i++)
                    if (st.ry >> i & 1) now += 0.5 * std::log2(1 + std::pow((double)st.rot[i][0] + st.rot[i][1], 2));
                most = std::max(most, now);
            }
    }
    *left = now;
    return most;
}
