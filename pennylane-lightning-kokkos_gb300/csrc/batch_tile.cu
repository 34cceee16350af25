// batch_tile.cu — batches of complex64 circuits on tiles.
//
// Every circuit of the batch (StateVectorKokkos::applyOperation over its tape,
// its Pauli-sum expectation value, AdjointDiffKokkos.hpp:404-478) is compiled
// once into symbolic tile programs (tile_program.hpp), forward and backward.  A
// run fills in the numbers that depend on the parameters (k_batch_evals,
// k_batch_runs, k_batch_fill) and then launches pass p of all circuits together:
// a launch's CTAs take tiles of different circuits, so the large circuits'
// passes and the small circuits' sweeps fill the GPU side by side, and a circuit
// of up to 11 qubits is one CTA's work per pass.  States live in one buffer, in
// waves of circuits when they are too large together.
//
// 128 circuits of 8-20 qubits, 5-30 layers on one GB300: 105.3 -> 15.3 ms a run
// (the engine's register windows spilled, and its largest circuits streamed their
// states from memory at 15 % of its bandwidth, one 8-CTA cluster each), first run
// with compilation 142 -> 39 ms.
// It replaces the persistent engine (batch.cu) for complex64 batches without
// dense matrices; those and complex128 batches keep it.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <thread>

#include "batch_tile.cuh"
#include "tile_launch.cuh"
#include "window_host.cuh"

namespace plk {

using namespace tile;

namespace {

constexpr int kBR = 4, kBT = 11;          // register bits, largest tiles
constexpr int kBThreads = 1 << (kBT - kBR);
constexpr int kBCtasFwd = 8, kBCtasBwd = 4;
constexpr size_t kBBlob = 12288;
constexpr int kHChunk = 4096;             // amplitudes per CTA of the Hamiltonian kernel

struct Job { // one pass of one circuit
    uint64_t lam, hl;     // offsets in the state buffer (amplitudes)
    uint64_t prog;        // offset of the blob (bytes)
    uint32_t prog_bytes;
    int32_t T, nacc;
    int32_t first_pass;   // forward: starts from |0...0>
    int32_t last_pass;    // backward: leaves no states
    uint64_t part;        // partial sums: [accumulator][CTA]
    int32_t nctas;
};
struct Cta {
    int32_t job, tile0, ntiles, slot;
};
struct HCta { // a chunk of H lambda
    uint64_t lam, hl;
    uint32_t i0, n;
    int32_t term0, nterms;
};
struct JTerm {
    uint64_t part;
    int32_t nctas, ref;
    double coef;
};

// ------------------------------------------------------------------ numbers --
__device__ __forceinline__ void trig(const double *params, int pidx, double (&f)[5]) {
    f[0] = 1.0;
    f[1] = f[2] = f[3] = f[4] = 0.0;
    if (pidx >= 0) {
        const double t = params[pidx];
        sincos(0.5 * t, &f[2], &f[1]);
        sincos(t, &f[4], &f[3]);
    }
}
__device__ __forceinline__ double2 entry(const double2 *__restrict__ basis, int e, const double (&f)[5]) {
    double re = 0.0, im = 0.0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const double2 a = basis[5 * e + i];
        re = fma(f[i], a.x, re);
        im = fma(f[i], a.y, im);
    }
    return make_double2(re, im);
}

__global__ void k_batch_evals(const SymEval *__restrict__ evals, int n, const double2 *__restrict__ basis,
                              const double *__restrict__ params, double2 *__restrict__ pool) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SymEval e = evals[i];
    double f[5];
    trig(params, e.pidx, f);
    for (int k = 0; k < e.n; k++) pool[e.pool + k] = entry(basis, e.basis + k, f);
}

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double zabs(double2 a) { return sqrt(fma(a.x, a.x, a.y * a.y)); }
__device__ __forceinline__ double2 unit(double2 a) { return zscale(a, 1.0 / zabs(a)); }

// Runs of one-wire gates: product, split diag(b) [[c, -s], [s, c]] diag(a) with
// c >= 0, and the generators' coefficients in the frame of the run's sums (the
// run's start; X and Y after the phases a).
__global__ void k_batch_runs(const SymRun *__restrict__ runs, int n, const SymGate *__restrict__ gates,
                             const double2 *__restrict__ basis, const double *__restrict__ params,
                             double2 *__restrict__ pool, float2 *__restrict__ rot, double *__restrict__ refs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SymRun r = runs[i];
    const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
    double2 m[4] = {one, zero, zero, one};
    bool grads = false;
    auto step = [&](const SymGate &g) {
        double f[5];
        trig(params, g.pidx, f);
        double2 u[4], t[4];
#pragma unroll
        for (int k = 0; k < 4; k++) u[k] = entry(basis, g.basis + k, f);
#pragma unroll
        for (int k = 0; k < 4; k++) t[k] = zadd(zmul(u[k & 2], m[k & 1]), zmul(u[(k & 2) | 1], m[2 | (k & 1)]));
#pragma unroll
        for (int k = 0; k < 4; k++) m[k] = t[k];
    };
    for (int g = r.head; g >= 0; g = gates[g].next) {
        step(gates[g]);
        grads = grads || gates[g].ref[0] >= 0 || gates[g].ref[1] >= 0 || gates[g].ref[2] >= 0 || gates[g].ref[3] >= 0;
    }
    double2 a0 = one, a1 = one;
    if (r.type == RT_DIAG) {
        pool[r.pool_a] = m[0];
        pool[r.pool_a + 1] = m[3];
    } else {
        double c, s;
        double2 b0 = one, b1 = one;
        if (r.type == RT_RIGHT) { // [[c, -s], [s, c]] diag(a)
            c = zabs(m[0]);
            s = zabs(m[2]);
            if (c >= s) {
                a0 = unit(m[0]);
                s = fma(m[2].x, a0.x, m[2].y * a0.y);
                a1 = unit(m[3]);
            } else {
                a0 = unit(m[2]);
                c = fma(m[0].x, a0.x, m[0].y * a0.y);
                a1 = unit(zscale(m[1], -1.0));
                if (c < 0.0) {
                    c = -c;
                    s = -s;
                    a0 = zscale(a0, -1.0);
                    a1 = zscale(a1, -1.0);
                }
            }
        } else if (r.type == RT_LEFT) { // diag(b) [[c, -s], [s, c]]
            c = zabs(m[0]);
            s = zabs(m[1]);
            if (c >= s) {
                b0 = unit(m[0]);
                s = -fma(m[1].x, b0.x, m[1].y * b0.y);
                b1 = unit(m[3]);
            } else {
                b0 = unit(zscale(m[1], -1.0));
                c = fma(m[0].x, b0.x, m[0].y * b0.y);
                b1 = unit(m[2]);
                if (c < 0.0) {
                    c = -c;
                    s = -s;
                    b0 = zscale(b0, -1.0);
                    b1 = zscale(b1, -1.0);
                }
            }
        } else {
            c = zabs(m[0]);
            s = zabs(m[2]);
            if (c >= s) {
                b0 = unit(m[0]);
                b1 = s > 0.0 ? unit(m[2]) : one;
                a1 = zmul(unit(m[3]), zconj(b1));
            } else {
                b1 = unit(m[2]);
                b0 = c > 0.0 ? unit(m[0]) : one;
                a1 = zmul(unit(zscale(m[1], -1.0)), zconj(b0));
            }
        }
        rot[i] = make_float2((float)(s / (1.0 + c)), (float)s);
        if (r.pool_a >= 0) {
            pool[r.pool_a] = a0;
            pool[r.pool_a + 1] = a1;
        }
        if (r.pool_b >= 0) {
            pool[r.pool_b] = b0;
            pool[r.pool_b + 1] = b1;
        }
    }
    if (!grads) return;
    const double2 ph = zmul(a1, zconj(a0)); // X -> cos X + sin Y, Y -> cos Y - sin X
    m[0] = m[3] = one;
    m[1] = m[2] = zero;
    for (int gi = r.head; gi >= 0; gi = gates[gi].next) {
        const SymGate g = gates[gi];
        if (g.ref[0] >= 0 || g.ref[1] >= 0 || g.ref[2] >= 0 || g.ref[3] >= 0) {
            // W = m^dag (sum_k g_k sigma_k) m
            const double2 G[4] = {make_double2(g.g[0] + g.g[3], 0.0), make_double2(g.g[1], -g.g[2]),
                                  make_double2(g.g[1], g.g[2]), make_double2(g.g[0] - g.g[3], 0.0)};
            double2 q[4], w[4];
#pragma unroll
            for (int k = 0; k < 4; k++) q[k] = zadd(zmul(G[k & 2], m[k & 1]), zmul(G[(k & 2) | 1], m[2 | (k & 1)]));
#pragma unroll
            for (int k = 0; k < 4; k++)
                w[k] = zadd(zmul(zconj(m[k >> 1]), q[k & 1]), zmul(zconj(m[2 | (k >> 1)]), q[2 | (k & 1)]));
            const double x = 0.5 * (w[1].x + w[2].x), y = 0.5 * (w[2].y - w[1].y);
            if (g.ref[0] >= 0) refs[g.ref[0]] = 0.5 * (w[0].x + w[3].x);
            if (g.ref[3] >= 0) refs[g.ref[3]] = 0.5 * (w[0].x - w[3].x);
            if (g.ref[1] >= 0) refs[g.ref[1]] = fma(x, ph.x, -y * ph.y);
            if (g.ref[2] >= 0) refs[g.ref[2]] = fma(x, ph.y, y * ph.x);
        }
        step(g);
    }
}

// Tables (16 threads each), then rotations, controlled rotations and indexed
// phases, into the blobs.
__global__ void k_batch_fill(const SymTable *__restrict__ tables, int ntables, const SymFactor *__restrict__ factors,
                             const SymPatch *__restrict__ patches, int npatches, const uint64_t *__restrict__ pass_at,
                             const double2 *__restrict__ pool, const float2 *__restrict__ rot, unsigned char *blobs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntables * kMaxAmps) {
        const SymTable t = tables[i / kMaxAmps];
        const int j = i % kMaxAmps;
        double2 z = make_double2(1.0, 0.0);
        for (int k = t.first; k < t.first + t.count; k++) {
            const SymFactor f = factors[k];
            int e = 0;
            if (f.K < 0) e = __popc(j & f.mask) & 1;
            else
                for (int q = 0; q < f.K; q++) e |= (j >> f.reg[q] & 1) << q;
            z = zmul(z, pool[f.pool + e]);
        }
        reinterpret_cast<float2 *>(blobs + pass_at[t.pass] + t.off)[j] = make_float2((float)z.x, (float)z.y);
        return;
    }
    const int p = i - ntables * kMaxAmps;
    if (p >= npatches) return;
    const SymPatch q = patches[p];
    float *dst = reinterpret_cast<float *>(blobs + pass_at[q.pass] + q.off);
    if (q.kind == 0) {
        const float2 r = rot[q.src];
        dst[0] = r.x;
        dst[2] = r.y;
    } else if (q.kind == 1) {
        dst[0] = (float)pool[q.src].x;
        dst[2] = (float)pool[q.src + 1].x;
    } else {
        for (int k = 0; k < q.n; k++) {
            dst[2 * k] = (float)pool[q.src + k].x;
            dst[2 * k + 1] = (float)pool[q.src + k].y;
        }
    }
}

// -------------------------------------------------------------------- sweeps --
template <bool BWD>
__global__ void __launch_bounds__(kBThreads, BWD ? kBCtasBwd : kBCtasFwd)
    k_batch_tile(const Cta *__restrict__ ctas, const Job *__restrict__ jobs, float2 *states, unsigned char *blobs,
                 double *__restrict__ part) {
    extern __shared__ __align__(16) unsigned char batch_smem[];
    const Cta c = ctas[blockIdx.x];
    const Job j = jobs[c.job];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tile_bytes = 8u << j.T;
    unsigned char *L = batch_smem, *M = L + tile_bytes;
    unsigned char *prog = batch_smem + (BWD ? 2 : 1) * tile_bytes;
    float2 *acc = reinterpret_cast<float2 *>(prog + j.prog_bytes);
    float2 *row = acc + warp * j.nacc;
    for (uint32_t i = tid * 16; i < j.prog_bytes; i += blockDim.x * 16)
        *reinterpret_cast<uint4 *>(prog + i) = __ldcg(reinterpret_cast<const uint4 *>(blobs + j.prog + i));
    if (BWD)
        for (int i = lane; i < j.nacc; i += 32) row[i] = make_float2(0.0f, 0.0f);
    __syncthreads();
    const Pass ps(prog);
    const Buffers bf{states + j.lam, states + j.lam, states + j.hl, 0, 0, !BWD && j.first_pass, BWD && j.last_pass, false, 0, 0, 0};
    for (int t = 0; t < c.ntiles; t++) run_tile<AmpC64, kBR, BWD>(ps, bf, c.tile0 + t, j.T, L, M, row);
    if (BWD) {
        for (int i = tid; i < j.nacc; i += blockDim.x) {
            DF s = {0.0f, 0.0f};
            for (int w = 0; w < (int)blockDim.x / 32; w++) df_add(acc[w * j.nacc + i].x, acc[w * j.nacc + i].y, s.hi, s.lo);
            part[j.part + (size_t)i * j.nctas + c.slot] = df_result(s.hi, s.lo);
        }
    }
}

// H lambda of a chunk and its part of <lambda|H|lambda>: H = sum_w c_w P_w with
// (P v)[i] = i^ny (-1)^popcount((i ^ x) & z) v[i ^ x]
__global__ void __launch_bounds__(kThreads)
    k_batch_h(const HCta *__restrict__ ctas, const ETerm *__restrict__ terms, float2 *states, double *__restrict__ part) {
    __shared__ double sums[kThreads / 32];
    const HCta c = ctas[blockIdx.x];
    const float2 *lam = states + c.lam;
    EAcc<float> acc;
    constexpr int F = 4; // gathers issued together
    for (uint32_t i = c.i0 + threadIdx.x; i < c.i0 + c.n; i += kThreads) {
        const float2 li = lam[i];
        float2 hs = make_float2(0.0f, 0.0f);
        for (int k0 = 0; k0 < c.nterms; k0 += F) {
            float2 v[F];
#pragma unroll
            for (int u = 0; u < F; u++)
                if (k0 + u < c.nterms) v[u] = lam[i ^ terms[c.term0 + k0 + u].x];
#pragma unroll
            for (int u = 0; u < F; u++) {
                if (k0 + u >= c.nterms) break;
                const ETerm tm = terms[c.term0 + k0 + u];
                const int q = (tm.ny + 2 * (__popc((i ^ tm.x) & tm.z) & 1)) & 3;
                const float2 w = v[u];
                const float2 x = q == 0 ? w : (q == 1 ? mul_i(w) : (q == 2 ? cneg(w) : mul_mi(w)));
                hs = make_float2(hs.x + (float)tm.c * x.x, hs.y + (float)tm.c * x.y);
                acc.re_dot_scaled(tm.ch, tm.cl, li, x);
            }
        }
        states[c.hl + i] = hs;
    }
    const double s = acc.warp_sum();
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kThreads / 32; w++) t += sums[w];
        part[blockIdx.x] = t;
    }
}

// results: one warp per Jacobian slot, then one per circuit; fixed order
__global__ void k_batch_results(const int *__restrict__ first, const JTerm *__restrict__ terms, int nslots,
                                const double *__restrict__ refs, const double *__restrict__ part, double *__restrict__ jac,
                                const int2 *__restrict__ ev_range, int ncirc, const double *__restrict__ ev_part,
                                double *__restrict__ expval) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    auto warp_total = [](double a) {
#pragma unroll
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        return a;
    };
    if (w < nslots) {
        double t = 0.0;
        for (int k = first[w]; k < first[w + 1]; k++) {
            const JTerm q = terms[k];
            double a = 0.0;
            for (int b = lane; b < q.nctas; b += 32) a += part[q.part + b];
            a = warp_total(a);
            t += (q.ref >= 0 ? q.coef * refs[q.ref] : q.coef) * a;
        }
        if (lane == 0) jac[w] = t;
    } else if (w - nslots < ncirc) {
        const int c = w - nslots;
        double a = 0.0;
        for (int b = ev_range[c].x + lane; b < ev_range[c].y; b += 32) a += ev_part[b];
        a = warp_total(a);
        if (lane == 0) expval[c] = a;
    }
}

// ---------------------------------------------------------------- host side --
// the primitives of one op with symbolic entries
struct Basis { // of a (gate, adjoint, direction): first entry of each primitive
    std::vector<int> at;
};

struct Program { // one direction of one circuit
    TileProgram P;
    Symbols S;
};

struct Compiled {
    Program dir[2];
    bool ok = false;
};

// entries of a primitive in the order that SymEval / SymGate use
int entries_of(const Prim &p, cplx *e) {
    switch (p.kind) {
    case P_U1: std::copy(p.m, p.m + 4, e); return 4;
    case tile::P_DIAG: std::copy(p.d, p.d + (1 << p.K), e); return 1 << p.K;
    case P_PAR: std::copy(p.d, p.d + 2, e); return 2;
    case P_CRY:
        e[0] = p.c;
        e[1] = p.s;
        return 2;
    default: return 0;
    }
}

struct BasisTable {
    std::vector<double2> v; // five per entry
    std::map<int, Basis> of;
    int one = 0;            // entry of the constant 1

    // lower_op of x at angle t
    static bool lower(const XOp &x, int nq, double t, bool bwd, int slot, Lowered &L) {
        int64_t w[32];
        int nw = 0;
        if (x.gate == PLK_GATE_MULTIRZ)
            for (int q : x.mrz_wires) w[nw++] = q;
        else
            for (; nw < x.K; nw++) w[nw] = x.wires[nw];
        plk_op op;
        std::memset(&op, 0, sizeof(op));
        op.gate = x.gate;
        op.num_wires = nw;
        op.adjoint = x.inv;
        op.num_params = x.pidx >= 0 ? 1 : 0;
        op.wires = w;
        op.params = &t;
        L.v.clear();
        if (!lower_op(op, nq, slot, L)) return false;
        if (bwd) invert(L.v);
        return true;
    }

    static int key(const XOp &x, bool bwd) { return (x.gate * 2 + x.inv) * 2 + bwd; }

    // fits every entry's five coefficients from five angles
    bool add(const XOp &x, int nq, bool bwd) {
        if (of.count(key(x, bwd))) return true;
        static const double th[5] = {0.37, 1.61, 2.83, 4.07, 5.51};
        double inv[5][10];
        for (int k = 0; k < 5; k++) {
            trig5(th[k], inv[k]);
            for (int c = 0; c < 5; c++) inv[k][5 + c] = c == k;
        }
        for (int c = 0; c < 5; c++) {
            int piv = c;
            for (int r = c + 1; r < 5; r++)
                if (std::fabs(inv[r][c]) > std::fabs(inv[piv][c])) piv = r;
            for (int j = 0; j < 10; j++) std::swap(inv[c][j], inv[piv][j]);
            const double d = inv[c][c];
            for (int j = 0; j < 10; j++) inv[c][j] /= d;
            for (int r = 0; r < 5; r++)
                if (r != c) {
                    const double f = inv[r][c];
                    for (int j = 0; j < 10; j++) inv[r][j] -= f * inv[c][j];
                }
        }
        std::vector<std::vector<cplx>> val(5);
        Basis b;
        Lowered L;
        for (int k = 0; k < 5; k++) {
            if (!lower(x, nq, th[k], bwd, -1, L)) return false;
            b.at.clear();
            for (const Prim &p : L.v) {
                cplx e[8];
                const int n = entries_of(p, e);
                b.at.push_back((int)(v.size() / 5 + val[k].size()));
                val[k].insert(val[k].end(), e, e + n);
            }
        }
        for (size_t e = 0; e < val[0].size(); e++)
            for (int i = 0; i < 5; i++) {
                cplx a = 0;
                for (int k = 0; k < 5; k++) a += inv[i][5 + k] * val[k][e];
                if (x.pidx < 0) a = i == 0 ? val[0][e] : cplx(0);
                v.push_back(make_double2(std::fabs(a.real()) < 1e-15 ? 0.0 : a.real(),
                                         std::fabs(a.imag()) < 1e-15 ? 0.0 : a.imag()));
            }
        of[key(x, bwd)] = b;
        return true;
    }
};

// Every index that the filling kernels follow, within one program.
bool check_symbols(const Program &p) {
    const Symbols &S = p.S;
    const int np = S.npool, ng = (int)S.gates.size(), nr = (int)S.runs.size();
    auto in_pool = [&](int at, int n) { return at >= 0 && at + n <= np; };
    for (const SymGate &g : S.gates) {
        if (g.next >= ng) return false;
        for (int r : g.ref)
            if (r >= S.nrefs) return false;
    }
    for (const SymRun &r : S.runs)
        if (r.head < 0 || r.head >= ng || (r.pool_a >= 0 && !in_pool(r.pool_a, 2)) || (r.pool_b >= 0 && !in_pool(r.pool_b, 2)))
            return false;
    for (const SymEval &e : S.evals)
        if (!in_pool(e.pool, e.n)) return false;
    for (const SymFactor &f : S.factors)
        if (f.K > 3 || !in_pool(f.pool, f.K < 0 ? 2 : 1 << f.K)) return false;
    auto room = [&](int pass, uint32_t off, size_t n) {
        return pass >= 0 && pass < (int)p.P.passes.size() && off + n <= p.P.passes[pass].blob.size();
    };
    for (const SymTable &t : S.tables)
        if (!room(t.pass, t.off, sizeof(float2) * kMaxAmps) || t.off % 8 || t.first < 0 || t.count < 0 ||
            (size_t)(t.first + t.count) > S.factors.size())
            return false;
    for (const SymPatch &q : S.patches) {
        if (!room(q.pass, q.off, q.kind == 2 ? sizeof(float2) * q.n : 16) || q.off % 4) return false;
        if (q.kind == 0 ? (q.src < 0 || q.src >= nr) : !in_pool(q.src, q.n)) return false;
    }
    return true;
}

bool compile_circuit(const BatchCircuit &c, const BasisTable &bt, Compiled &out) {
    Options o;
    o.T = kBT;
    o.R = kBR;
    o.low = 3;
    o.amp_bytes = 8;
    o.max_blob = kBBlob;
    const std::vector<XOp> &ops = *c.ops;
    for (int dir = 0; dir < 2; dir++) {
        const bool bwd = dir == 1;
        Program &pr = out.dir[dir];
        Compiler k(c.nq, bwd, o, &pr.S);
        Lowered L;
        // ops before the first trainable op do not change the Jacobian (the
        // reference loop ends there too, AdjointDiffKokkos.hpp:447)
        int from = 0;
        const int n = (int)ops.size();
        if (bwd)
            while (from < n && ops[from].slot < 0) from++;
        auto put = [&](const XOp &x) {
            // any angle will do: the program holds no numbers
            if (!BasisTable::lower(x, c.nq, 0.7, bwd, bwd ? x.slot : -1, L)) return false;
            const Basis &b = bt.of.at(BasisTable::key(x, bwd));
            for (size_t i = 0; i < L.v.size(); i++) {
                L.v[i].sbasis = b.at[i];
                L.v[i].spidx = x.pidx;
            }
            k.add(L.v);
            return true;
        };
        if (!bwd) {
            for (int i = 0; i < n; i++)
                if (!put(ops[i])) return false;
            // something to write the state with
            Prim p;
            p.kind = tile::P_DIAG;
            p.K = 1;
            p.d[0] = p.d[1] = 1;
            p.sbasis = bt.one;
            if (n == 0) k.add({p});
        } else {
            for (int i = n - 1; i >= from; i--)
                if (!put(ops[i])) return false;
        }
        if (!k.compile(pr.P)) return false;
        for (const TilePass &ps : pr.P.passes)
            if (!check_pass(ps, c.nq, 8, pr.P.nacc)) return false;
        if (!check_symbols(pr)) return false;
    }
    return true;
}

struct LaunchItem {
    int kind; // 0 forward, 1 H, 2 backward
    int cta0, nctas, threads;
    size_t smem;
};

} // namespace

struct BatchTiles {
    int device = 0;
    void *block = nullptr; // what the pointers below point into
    SymEval *evals = nullptr;
    SymRun *runs = nullptr;
    SymGate *gates = nullptr;
    SymTable *tables = nullptr;
    SymFactor *factors = nullptr;
    SymPatch *patches = nullptr;
    uint64_t *pass_at = nullptr;
    double2 *basis = nullptr, *pool = nullptr;
    float2 *rot = nullptr;
    double *refs = nullptr;
    unsigned char *blobs = nullptr;
    Job *jobs = nullptr;
    Cta *ctas = nullptr;
    HCta *hctas = nullptr;
    ETerm *terms = nullptr;
    float2 *states = nullptr;
    double *part = nullptr, *ev_part = nullptr;
    int *jfirst = nullptr;
    int2 *ev_range = nullptr; // chunks of the Hamiltonian kernel by circuit
    JTerm *jterms = nullptr;
    int nevals = 0, nruns = 0, ntables = 0, npatches = 0, nslots = 0, ncirc = 0;
    std::vector<LaunchItem> launches;
    ~BatchTiles() {
        if (block) cudaFree(block);
    }
};

void batch_tiles_destroy(BatchTiles *t) { delete t; }

int batch_tiles_launches(const BatchTiles *t) { return (int)t->launches.size() + 4; }

namespace {

// One allocation for everything a batch has on the device, and one copy for what is
// small: 22 allocations and 16 copies took 40 us more of the 0.6-0.8 ms of a small
// batch's first run, and as much of its 0.3 ms of destruction.
class Block {
  public:
    template <class V> void upload(V *&dst, const std::vector<V> &src) {
        parts_.push_back({reinterpret_cast<void **>(&dst), src.data(), src.size() * sizeof(V), 0});
    }
    template <class V> void reserve(V *&dst, size_t n) {
        parts_.push_back({reinterpret_cast<void **>(&dst), nullptr, n * sizeof(V), 0});
    }
    // allocates, points every dst into the block and queues the copies (the sources
    // stay until the stream is waited for)
    int commit(void *&block, cudaStream_t st) {
        constexpr size_t kSmall = 65536;
        auto place = [&](bool small, size_t at) {
            for (Part &p : parts_)
                if ((p.src && p.bytes <= kSmall) == small) {
                    p.at = at;
                    at += (std::max<size_t>(p.bytes, 1) + 255) & ~(size_t)255;
                }
            return at;
        };
        const size_t front = place(true, 0), total = place(false, front);
        PLK_CUDA(cudaMalloc(&block, std::max<size_t>(total, 256)));
        host_.assign(front, 0);
        for (Part &p : parts_) {
            unsigned char *dst = static_cast<unsigned char *>(block) + p.at;
            *p.dst = dst;
            if (!p.src || !p.bytes) continue;
            if (p.bytes <= kSmall) std::memcpy(host_.data() + p.at, p.src, p.bytes);
            else PLK_CUDA(cudaMemcpyAsync(dst, p.src, p.bytes, cudaMemcpyHostToDevice, st));
        }
        if (front) PLK_CUDA(cudaMemcpyAsync(block, host_.data(), front, cudaMemcpyHostToDevice, st));
        return PLK_OK;
    }

  private:
    struct Part {
        void **dst;
        const void *src;
        size_t bytes, at;
    };
    std::vector<Part> parts_;
    std::vector<unsigned char> host_;
};

int build(BatchTiles *t, const std::vector<BatchCircuit> &circs, const BasisTable &bt, std::vector<Compiled> &cc,
          cudaStream_t st) {
    DeviceCtx *d = nullptr;
    PLK_TRY(device_ctx(t->device, &d));
    // one list of symbols: offsets of each program's pieces
    std::vector<SymEval> evals;
    std::vector<SymRun> runs;
    std::vector<SymGate> gates;
    std::vector<SymTable> tables;
    std::vector<SymFactor> factors;
    std::vector<SymPatch> patches;
    std::vector<uint64_t> pass_at;
    std::vector<unsigned char> blobs;
    std::vector<int> pass0(2 * circs.size()), ref0(2 * circs.size());
    int npool = 0, nrefs = 0;
    for (size_t ci = 0; ci < circs.size(); ci++)
        for (int dir = 0; dir < 2; dir++) {
            const Program &p = cc[ci].dir[dir];
            const Symbols &S = p.S;
            const int g0 = (int)gates.size(), r0 = (int)runs.size(), f0 = (int)factors.size(), p0 = (int)pass_at.size();
            pass0[2 * ci + dir] = p0;
            ref0[2 * ci + dir] = nrefs;
            for (SymGate g : S.gates) {
                if (g.next >= 0) g.next += g0;
                for (int &r : g.ref)
                    if (r >= 0) r += nrefs;
                gates.push_back(g);
            }
            for (SymRun r : S.runs) {
                r.head += g0;
                if (r.pool_a >= 0) r.pool_a += npool;
                if (r.pool_b >= 0) r.pool_b += npool;
                runs.push_back(r);
            }
            for (SymEval e : S.evals) {
                e.pool += npool;
                evals.push_back(e);
            }
            for (SymFactor f : S.factors) {
                f.pool += npool;
                factors.push_back(f);
            }
            for (SymTable q : S.tables) {
                q.pass += p0;
                q.first += f0;
                tables.push_back(q);
            }
            for (SymPatch q : S.patches) {
                q.pass += p0;
                q.src += q.kind == 0 ? r0 : npool;
                patches.push_back(q);
            }
            npool += S.npool;
            nrefs += S.nrefs;
            for (const TilePass &ps : p.P.passes) {
                pass_at.push_back(blobs.size());
                blobs.insert(blobs.end(), ps.blob.begin(), ps.blob.end());
            }
        }
    // waves of circuits whose states fit the budget, large circuits first
    std::vector<int> order(circs.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return circs[a].nq > circs[b].nq; });
    size_t fr = 0, tot = 0;
    PLK_CUDA(cudaMemGetInfo(&fr, &tot));
    const uint64_t budget = std::min<uint64_t>((uint64_t)16 << 30, fr / 2) / sizeof(float2);
    std::vector<std::vector<int>> waves;
    std::vector<uint64_t> state_at(circs.size());
    uint64_t used = 0, most = 0;
    for (int i : order) {
        const uint64_t n = 2ull << circs[i].nq;
        if (waves.empty() || used + n > budget) {
            waves.emplace_back();
            used = 0;
        }
        waves.back().push_back(i);
        state_at[i] = used;
        used += n;
        most = std::max(most, used);
    }
    // jobs, and each launch's CTAs: pass p of all circuits of a wave
    std::vector<Job> jobs;
    std::vector<Cta> ctas;
    std::vector<HCta> hctas;
    std::vector<ETerm> terms;
    std::vector<int> term0(circs.size());
    for (size_t i = 0; i < circs.size(); i++) {
        term0[i] = (int)terms.size();
        terms.insert(terms.end(), circs[i].terms->begin(), circs[i].terms->end());
    }
    std::vector<std::vector<std::pair<int, int>>> job_of(2 * circs.size()); // (job, first accumulator)
    std::vector<int2> ev_range(circs.size());
    uint64_t npart = 0;
    auto sweeps = [&](const std::vector<int> &wave, int dir) {
        size_t most_passes = 0;
        for (int i : wave) most_passes = std::max(most_passes, cc[i].dir[dir].P.passes.size());
        for (size_t p = 0; p < most_passes; p++) {
            uint64_t total = 0; // tiles of the launch
            for (int i : wave)
                if (p < cc[i].dir[dir].P.passes.size()) total += 1ull << (circs[i].nq - cc[i].dir[dir].P.T);
            // a few tiles per CTA share the program's load, when there are CTAs enough
            const uint64_t room = (uint64_t)d->sm_count * (dir ? kBCtasBwd : kBCtasFwd) * 2;
            const int each = (int)std::min<uint64_t>(8, std::max<uint64_t>(1, total / room));
            // by threads per tile: 128, 64, 32
            for (int th = kBThreads; th >= 32; th /= 2) {
                LaunchItem l{dir ? 2 : 0, (int)ctas.size(), 0, th, 0};
                for (int i : wave) {
                    const TileProgram &P = cc[i].dir[dir].P;
                    if (p >= P.passes.size() || std::max(32, 1 << (P.T - P.R)) != th) continue;
                    const TileHdr &h = *reinterpret_cast<const TileHdr *>(P.passes[p].blob.data());
                    const int ntiles = 1 << (circs[i].nq - P.T);
                    Job j;
                    std::memset((void *)&j, 0, sizeof(j));
                    j.lam = state_at[i];
                    j.hl = state_at[i] + (1ull << circs[i].nq);
                    j.prog = pass_at[pass0[2 * i + dir] + p];
                    j.prog_bytes = h.bytes;
                    j.T = P.T;
                    j.nacc = h.nacc;
                    j.first_pass = p == 0;
                    j.last_pass = p + 1 == (int)P.passes.size();
                    j.nctas = (ntiles + each - 1) / each;
                    j.part = npart;
                    npart += (uint64_t)h.nacc * j.nctas;
                    job_of[2 * i + dir].push_back({(int)jobs.size(), h.acc0});
                    for (int k = 0; k < j.nctas; k++)
                        ctas.push_back(Cta{(int)jobs.size(), k * each, std::min(each, ntiles - k * each), k});
                    jobs.push_back(j);
                    l.smem = std::max(l.smem, smem_bytes(8, dir == 1, P.T, h.bytes, h.nacc, th));
                }
                l.nctas = (int)ctas.size() - l.cta0;
                if (l.nctas) t->launches.push_back(l);
            }
        }
    };
    for (const auto &wave : waves) {
        sweeps(wave, 0);
        LaunchItem l{1, (int)hctas.size(), 0, kThreads, 0};
        for (int i : wave) {
            const uint32_t n = 1u << circs[i].nq;
            ev_range[i].x = (int)hctas.size();
            for (uint32_t at = 0; at < n; at += kHChunk)
                hctas.push_back(HCta{state_at[i], state_at[i] + n, at, std::min<uint32_t>(kHChunk, n - at), term0[i],
                                     (int)circs[i].terms->size()});
            ev_range[i].y = (int)hctas.size();
        }
        l.nctas = (int)hctas.size() - l.cta0;
        t->launches.push_back(l);
        sweeps(wave, 1);
    }
    // Jacobian: terms by slot
    int nslots = 0;
    for (const BatchCircuit &c : circs) nslots = std::max(nslots, c.jac0 + c.ntp);
    std::vector<int> first(nslots + 1, 0);
    std::vector<std::pair<int, JTerm>> list;
    for (size_t i = 0; i < circs.size(); i++) {
        const Program &p = cc[i].dir[1];
        const double share = (double)(1 << (p.P.T - p.P.R)) / std::max(32, 1 << (p.P.T - p.P.R));
        const auto &jo = job_of[2 * i + 1];
        size_t k = 0;
        for (const JacTerm &q : p.P.jac) { // in pass order
            while (k + 1 < jo.size() && q.acc >= jo[k + 1].second) k++;
            while (k > 0 && q.acc < jo[k].second) k--;
            const Job &j = jobs[jo[k].first];
            if (q.acc - jo[k].second >= j.nacc || q.slot < 0 || q.slot >= circs[i].ntp)
                PLK_FAIL(PLK_ERR_UNSUPPORTED, "internal: batch program check failed");
            JTerm v;
            v.part = j.part + (uint64_t)(q.acc - jo[k].second) * j.nctas;
            v.nctas = j.nctas;
            v.ref = q.ref >= 0 ? q.ref + ref0[2 * i + 1] : -1;
            v.coef = q.coef * share;
            list.push_back({circs[i].jac0 + q.slot, v});
            first[circs[i].jac0 + q.slot + 1]++;
        }
    }
    for (int s = 0; s < nslots; s++) first[s + 1] += first[s];
    std::vector<JTerm> jterms(list.size());
    {
        std::vector<int> next(first.begin(), first.end() - 1);
        for (const auto &e : list) jterms[next[e.first]++] = e.second;
    }
    t->nevals = (int)evals.size();
    t->nruns = (int)runs.size();
    t->ntables = (int)tables.size();
    t->npatches = (int)patches.size();
    t->nslots = nslots;
    t->ncirc = (int)circs.size();
    Block b;
    b.upload(t->evals, evals);
    b.upload(t->runs, runs);
    b.upload(t->gates, gates);
    b.upload(t->tables, tables);
    b.upload(t->factors, factors);
    b.upload(t->patches, patches);
    b.upload(t->pass_at, pass_at);
    b.upload(t->basis, bt.v);
    b.upload(t->blobs, blobs);
    b.upload(t->jobs, jobs);
    b.upload(t->ctas, ctas);
    b.upload(t->hctas, hctas);
    b.upload(t->terms, terms);
    b.upload(t->jfirst, first);
    b.upload(t->jterms, jterms);
    b.upload(t->ev_range, ev_range);
    b.reserve(t->pool, npool);
    b.reserve(t->rot, runs.size());
    b.reserve(t->refs, nrefs);
    b.reserve(t->states, most);
    b.reserve(t->part, npart);
    b.reserve(t->ev_part, hctas.size());
    PLK_TRY(b.commit(t->block, st));
    PLK_CUDA(cudaFuncSetAttribute(k_batch_tile<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem_bytes(8, false, kBT, kBBlob, 0, kBThreads)));
    PLK_CUDA(cudaFuncSetAttribute(k_batch_tile<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem_bytes(8, true, kBT, kBBlob, 2 * kMaxAcc, kBThreads)));
    PLK_CUDA(cudaStreamSynchronize(st));
    return PLK_OK;
}

} // namespace

int batch_tiles_create(const std::vector<BatchCircuit> &circs, int device, cudaStream_t st, BatchTiles **out) {
    *out = nullptr;
    BasisTable bt;
    bt.v.push_back(make_double2(1.0, 0.0)); // the constant 1, twice (a diagonal on one bit)
    for (int k = 0; k < 9; k++) bt.v.push_back(make_double2(k == 4 ? 1.0 : 0.0, 0.0));
    for (const BatchCircuit &c : circs)
        for (const XOp &x : *c.ops)
            for (bool bwd : {false, true})
                if (x.gate == PLK_GATE_MATRIX || !bt.add(x, c.nq, bwd)) return PLK_OK;
    // circuits are independent: compiled by a few threads
    std::vector<Compiled> cc(circs.size());
    std::atomic<size_t> next{0};
    std::atomic<bool> ok{true};
    auto work = [&]() {
        for (;;) {
            const size_t i = next.fetch_add(1);
            if (i >= circs.size() || !ok.load()) return;
            try {
                if (!compile_circuit(circs[i], bt, cc[i])) ok.store(false);
            } catch (...) {
                ok.store(false);
            }
        }
    };
    // by ops, not by circuits: an op takes some 2 us to compile, both ways, a thread
    // 20-30 us to start (16 circuits of 12 qubits and 100 layers, first run: 2 threads
    // 32.5 ms, 16 threads 14.2; two circuits of 70 ops 0.58 ms with one, 0.65 with two)
    size_t nops = 0;
    for (const BatchCircuit &c : circs) nops += c.ops->size();
    const unsigned n =
        std::min<size_t>({std::max(1u, std::thread::hardware_concurrency()), 16, circs.size(), 1 + nops / 1024});
    std::vector<std::thread> pool;
    for (unsigned k = 1; k < n; k++) {
        try {
            pool.emplace_back(work);
        } catch (...) {
            break; // fewer threads
        }
    }
    work();
    for (auto &th : pool) th.join();
    if (!ok.load()) return PLK_OK;
    BatchTiles *t = new BatchTiles();
    t->device = device;
    const int rc = build(t, circs, bt, cc, st);
    if (rc != PLK_OK) {
        cudaStreamSynchronize(st);
        delete t;
        if (rc != PLK_ERR_OUT_OF_MEMORY) return rc;
        // The engine keeps no circuit's state for longer than it runs, no programs
        // (some hundred KB per circuit) and no partial sums by tile: small circuits
        // need a fraction of this there.  What it cannot allocate it reports.
        cudaGetLastError();
        set_error(std::string());
        return PLK_OK;
    }
    *out = t;
    return PLK_OK;
}

int batch_tiles_enqueue(BatchTiles *t, const double *d_params, double *d_expval, double *d_jac, cudaStream_t st) {
    if (t->nevals) k_batch_evals<<<(t->nevals + 127) / 128, 128, 0, st>>>(t->evals, t->nevals, t->basis, d_params, t->pool);
    if (t->nruns)
        k_batch_runs<<<(t->nruns + 127) / 128, 128, 0, st>>>(t->runs, t->nruns, t->gates, t->basis, d_params, t->pool,
                                                            t->rot, t->refs);
    const int fills = t->ntables * kMaxAmps + t->npatches;
    if (fills)
        k_batch_fill<<<(fills + 127) / 128, 128, 0, st>>>(t->tables, t->ntables, t->factors, t->patches, t->npatches,
                                                         t->pass_at, t->pool, t->rot, t->blobs);
    PLK_CHECK_LAUNCH();
    for (const LaunchItem &l : t->launches) {
        if (l.kind == 0)
            k_batch_tile<false><<<l.nctas, l.threads, l.smem, st>>>(t->ctas + l.cta0, t->jobs, t->states, t->blobs, t->part);
        else if (l.kind == 1)
            k_batch_h<<<l.nctas, l.threads, 0, st>>>(t->hctas + l.cta0, t->terms, t->states, t->ev_part + l.cta0);
        else
            k_batch_tile<true><<<l.nctas, l.threads, l.smem, st>>>(t->ctas + l.cta0, t->jobs, t->states, t->blobs, t->part);
        PLK_CHECK_LAUNCH();
    }
    const int warps = t->nslots + t->ncirc;
    k_batch_results<<<(warps + 7) / 8, 256, 0, st>>>(t->jfirst, t->jterms, t->nslots, t->refs, t->part, d_jac, t->ev_range,
                                                    t->ncirc, t->ev_part, d_expval);
    PLK_CHECK_LAUNCH();
    return PLK_OK;
}

} // namespace plk
