// Runs tile programs (csrc/tile_program.hpp) on the CPU, thread by thread, in
// double precision: the same blobs, slot maps, steps and sums that
// tile_kernels.cuh follows on the GPU.  Built as a shared library by
// tests/test_tile_program_cpu.py and compared there with the oracle.
#include <complex>
#include <cstdio>
#include <vector>

#include "tile_program.hpp"

using namespace plk::tile;
using C = std::complex<double>;

namespace {

struct Emu {
    const unsigned char *b;
    const TileHdr *h;
    int amp;
    C entry(uint32_t e) const {
        const float *f = reinterpret_cast<const float *>(b + h->off_tab + (size_t)e * amp);
        return amp == 8 ? C(f[0], f[1]) : C((double)f[0] + f[2], (double)f[1] + f[3]);
    }
    double gen(uint32_t e) const { return reinterpret_cast<const float *>(b + h->off_tab)[e]; }
};

double imdot(C h, C v) { return h.real() * v.imag() - h.imag() * v.real(); }

int slot_of(const TileRound &m, int t, int j, uint32_t ev, int amp, const TileHdr &h) {
    uint32_t o = m.lo[t & 31] ^ m.hi[t >> 5] ^ m.xorc ^ ev;
    for (int i = 0; i < h.R; i++)
        if (j >> i & 1) o ^= m.rcol[i];
    if (o % amp || o / amp >= (1u << h.T)) return -1;
    return (int)(o / amp);
}

uint32_t index_of(const TileIndex &x, int t, int j, int R) {
    uint32_t g = x.lo[t & 31] ^ x.hi[t >> 5] ^ x.c;
    for (int i = 0; i < R; i++)
        if (j >> i & 1) g ^= x.r[i];
    return g;
}

} // namespace

// Sweeps lam (and hl when bwd) in place; slot[i] >= 0: op i's Jacobian slot.
// Returns the number of passes, negative on a failed check.
extern "C" int tile_emulate(int nq, int T, int R, int low, int amp, int bwd, const plk_op *ops, int nops,
                            const int64_t *slot, C *lam, C *hl, double *jac, int nslots, int *rounds) {
    Options o;
    o.T = T;
    o.R = R;
    o.low = low;
    o.amp_bytes = amp;
    Compiler c(nq, bwd != 0, o);
    for (int k = 0; k < nops; k++) {
        const int i = bwd ? nops - 1 - k : k;
        Lowered L;
        if (!lower_op(ops[i], nq, bwd ? (int)slot[i] : -1, L)) return -100;
        if (bwd) invert(L.v);
        c.add(L.v);
    }
    TileProgram P;
    if (!c.compile(P)) return -101;
    std::vector<double> acc(P.nacc + 1, 0.0);
    *rounds = 0;
    for (const TilePass &ps : P.passes) {
        if (!check_pass(ps, nq, amp, P.nacc)) return -102;
        Emu e{ps.blob.data(), reinterpret_cast<const TileHdr *>(ps.blob.data()), amp};
        const TileHdr &h = *e.h;
        const int N = 1 << h.T, A = 1 << h.R, nth = N / A;
        *rounds += h.nrounds;
        if (h.bytes > o.max_blob) return -102;
        const TileRound *RR = reinterpret_cast<const TileRound *>(e.b + h.off_rounds);
        const TileStage *S = reinterpret_cast<const TileStage *>(e.b + h.off_stages);
        const TileEvent *E = reinterpret_cast<const TileEvent *>(e.b + h.off_events);
        const TileIndex *X = reinterpret_cast<const TileIndex *>(e.b + h.off_index);
        for (uint32_t tile = 0; tile < (1u << (nq - h.T)); tile++) {
            uint32_t base = tile;
            for (int k = 0; k < h.T; k++) {
                const uint32_t lo = base & ((1u << h.gpos[k]) - 1);
                base = ((base ^ lo) << 1) | lo;
            }
            std::vector<C> L(N), M(N), v(N), w(N); // slots; registers [thread][j]
            std::vector<int> seen(N, 0), where(N);
            uint32_t ev = 0;
            for (int r = 0; r < h.nrounds; r++) {
                const TileRound &q = RR[r];
                uint32_t gev = 0;
                for (int k = 0; k < q.nev; k++)
                    if (base >> E[q.ev0 + k].bit & 1) ev ^= E[q.ev0 + k].mask, gev ^= E[q.ev0 + k].gmask;
                std::fill(seen.begin(), seen.end(), 0);
                std::vector<uint32_t> used;
                for (int t = 0; t < nth; t++)
                    for (int j = 0; j < A; j++) {
                        const int s = slot_of(q, t, j, ev, amp, h);
                        if (s < 0 || seen[s]++) return -104;
                        where[t * A + j] = s;
                        if (r == 0) {
                            const uint32_t g = base ^ gev ^ index_of(X[h.load_idx], t, j, h.R);
                            if (g >> nq) return -103;
                            used.push_back(g);
                            v[t * A + j] = lam[g];
                            if (bwd) w[t * A + j] = hl[g];
                        } else {
                            v[t * A + j] = L[s];
                            if (bwd) w[t * A + j] = M[s];
                        }
                    }
                std::sort(used.begin(), used.end());
                if (std::unique(used.begin(), used.end()) != used.end()) return -103;
                for (int t = 0; t < nth; t++) {
                    C *V = &v[t * A], *W = &w[t * A];
                    auto full = [&](int j) { return base ^ index_of(X[q.idx], t, j, h.R); };
                    for (int k = 0; k < q.nstages; k++) {
                        const TileStage &st = S[q.stage0 + k];
                        if (st.table & 1) {
                            int a = st.acc_z;
                            for (int m = 0; m < kMaxAmps; m++)
                                if (st.zsel >> m & 1) {
                                    for (int j = 0; j < A; j++)
                                        acc[h.acc0 + a] += imdot(W[j], V[j]) * (__builtin_parity(j & m) ? -1 : 1);
                                    a++;
                                }
                        }
                        if (st.table & 2)
                            for (int j = 0; j < A; j++) {
                                V[j] *= e.entry(st.tab + j);
                                W[j] *= e.entry(st.tab + j);
                            }
                        for (int b = 0; b < h.R; b++) {
                            if (!(st.ry >> b & 1)) continue;
                            const double tt = (double)st.rot[b][0] + st.rot[b][1];
                            const double ss = (double)st.rot[b][2] + st.rot[b][3];
                            for (int j = 0; j < A; j++) {
                                const int j1 = j | 1 << b;
                                if (j == j1) continue;
                                C &x = V[j], &y = V[j1], &hx = W[j], &hy = W[j1];
                                if (st.acc_y[b] >= 0)
                                    acc[h.acc0 + st.acc_y[b]] += (std::conj(hy) * x).real() - (std::conj(hx) * y).real();
                                if (st.acc_x[b] >= 0) acc[h.acc0 + st.acc_x[b]] += imdot(hx, y) + imdot(hy, x);
                                for (int z = 0; z < 2; z++) {
                                    C &p = z ? hx : x, &u = z ? hy : y;
                                    if (amp == 16) { // complex128: [[1, -t], [t, 1]]
                                        const C p0 = p;
                                        p -= tt * u;
                                        u += tt * p0;
                                    } else {
                                        p -= tt * u;
                                        u += ss * p;
                                        p -= tt * u;
                                    }
                                }
                            }
                        }
                        if (st.special == TS_CRY) {
                            const uint32_t gi = st.cmask ? full(0) : 0;
                            if ((gi & st.cmask) != st.cval) continue;
                            const double cc = (double)st.coef[0] + st.coef[1], ss = (double)st.coef[2] + st.coef[3];
                            for (int j = 0; j < A; j++) {
                                const int j1 = j | 1 << st.bit;
                                if (j == j1 || !(st.jact >> j & 1)) continue;
                                const C x = V[j], y = V[j1], hx = W[j], hy = W[j1];
                                if (st.sacc >= 0)
                                    acc[h.acc0 + st.sacc] += (std::conj(hy) * x).real() - (std::conj(hx) * y).real();
                                V[j] = cc * x - ss * y;
                                V[j1] = ss * x + cc * y;
                                W[j] = cc * hx - ss * hy;
                                W[j1] = ss * hx + cc * hy;
                            }
                        } else if (st.special != TS_NONE) {
                            for (int j = 0; j < A; j++) {
                                uint32_t f = 0;
                                double g = 0;
                                if (st.special == TS_PAR) {
                                    f = __builtin_parity(full(j) & st.cmask);
                                    g = f ? -1 : 1;
                                } else {
                                    for (int i = 0; i < st.K; i++) f |= (full(j) >> (st.cmask >> (5 * i) & 31) & 1) << i;
                                    if (st.sacc >= 0) g = e.gen(st.gtab + f);
                                }
                                if (st.sacc >= 0) acc[h.acc0 + st.sacc] += g * imdot(W[j], V[j]);
                                V[j] *= e.entry(st.stab + f);
                                W[j] *= e.entry(st.stab + f);
                            }
                        }
                    }
                }
                for (int i = 0; i < N; i++) {
                    L[where[i]] = v[i];
                    M[where[i]] = w[i];
                }
            }
            uint32_t gev = 0;
            for (int k = h.ev_store0; k < h.nev; k++)
                if (base >> E[k].bit & 1) gev ^= E[k].gmask;
            std::vector<uint32_t> used;
            for (int t = 0; t < nth; t++)
                for (int j = 0; j < A; j++) {
                    const uint32_t g = base ^ gev ^ index_of(X[h.store_idx], t, j, h.R);
                    if (g >> nq) return -105;
                    used.push_back(g);
                    lam[g] = v[t * A + j];
                    if (bwd) hl[g] = w[t * A + j];
                }
            std::sort(used.begin(), used.end());
            if (std::unique(used.begin(), used.end()) != used.end()) return -105;
        }
    }
    for (int i = 0; i < nslots; i++) jac[i] = 0;
    for (const JacTerm &t : P.jac) {
        if (t.slot < 0 || t.slot >= nslots || t.acc < 0 || t.acc >= P.nacc) return -106;
        jac[t.slot] += t.coef * acc[t.acc];
    }
    return (int)P.passes.size();
}
