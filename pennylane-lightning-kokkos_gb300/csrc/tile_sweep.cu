// tile_sweep.cu — op lists and adjoint sweeps as tile programs.
//
// plk_apply_ops (StateVectorKokkos::applyOperation over a tape,
// StateVectorKokkos.hpp:585-676) and plk_adjoint_jacobian
// (AdjointDiffKokkos.hpp:404-478) compile their ops into passes over the state
// (tile_program.hpp) and launch one kernel per pass (tile_kernels.cuh).  The
// sweeps of several observables run in the same launches (gridDim.y), each on
// its own copy of lambda.  Op lists with dense matrices keep the register
// windows (windows.cu).
#include <algorithm>
#include <vector>

#include "gate_ops.cuh"
#include "sweep_cost.hpp"
#include "tile_launch.cuh"

namespace plk {

bool window_path_enabled();
int adjoint_gates(plk_state work, plk_state *hlambda, int32_t nobs, const plk_op *ops, int32_t nops,
                  const int64_t *trainable, int32_t ntp, double *jac);
int plan_generator(int gate, int nw, GatePlan &p);

namespace tile {

// jac[y][s] = sum over the slot's terms of coef * (the accumulator's sum over
// CTAs); one warp per slot, CTAs in lane-strided order, fixed pattern
__global__ void k_tile_jac(const double *__restrict__ part, int nblocks, int nacc_all, const int *__restrict__ first,
                           const int *__restrict__ term_acc, const double *__restrict__ term_coef, int nslots,
                           double *__restrict__ jac) {
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s >= nslots) return;
    const double *p = part + (size_t)blockIdx.y * nacc_all * nblocks;
    double t = 0.0;
    for (int k = first[s]; k < first[s + 1]; k++) {
        double a = 0.0;
        for (int b = lane; b < nblocks; b += 32) a += p[(size_t)term_acc[k] * nblocks + b];
#pragma unroll
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        t += term_coef[k] * a;
    }
    if (lane == 0) jac[(size_t)blockIdx.y * nslots + s] = t;
}

struct Shape {
    int R, threads, ctas;
};
static Shape shape(int dtype, bool bwd) {
    if (dtype == PLK_C64)
        return bwd ? Shape{kRegsC64Bwd, kThreadsC64Bwd, kCtasC64Bwd} : Shape{kRegsC64Fwd, kThreadsC64Fwd, kCtasC64Fwd};
    return bwd ? Shape{kRegsC128Bwd, kThreadsC128Bwd, kCtasC128Bwd}
               : Shape{kRegsC128Fwd, kThreadsC128Fwd, kCtasC128Fwd};
}

static int tile_bits(int nq, int dtype, bool bwd) {
    const Shape sh = shape(dtype, bwd);
    int T = sh.R;
    while ((1 << (T - sh.R)) < sh.threads) T++;
    return std::min(T, nq);
}

struct Word { // coeff i^ny (-1)^popcount(k & z) |k ^ x>
    uint32_t x, z;
    int ny;
    double coeff;
};

static Options options(int nq, int dtype, bool bwd) {
    Options o;
    o.T = tile_bits(nq, dtype, bwd);
    o.R = shape(dtype, bwd).R;
    o.amp_bytes = dtype == PLK_C64 ? 8 : 16;
    o.low = dtype == PLK_C64 ? 3 : 2; // 64-byte runs
    o.max_blob = kMaxBlob;
    return o;
}

static int check_program(const TileProgram &P, int amp_bytes) {
    for (const TilePass &p : P.passes)
        if (!check_pass(p, P.nq, amp_bytes, P.nacc)) PLK_FAIL(PLK_ERR_UNSUPPORTED, "internal: tile program check failed");
    for (const JacTerm &t : P.jac)
        if (t.acc < 0 || t.acc >= P.nacc) PLK_FAIL(PLK_ERR_UNSUPPORTED, "internal: tile program check failed");
    return PLK_OK;
}

// Runs P on nsweep (lambda, H lambda) pairs on stream st.  Backward, the
// Jacobian rows go to jac_host (row-major [nsweep][nslots]; synchronizes).
// words: H lambda of each sweep starts as that Pauli word on lam_src instead of
// what hl holds.
static int run(const TileProgram &P, int dtype, int device, cudaStream_t st, const void *const *lam_src,
               void *const *lam, void *const *hl, int nsweep, int nslots, double *jac_host,
               const Word *words = nullptr) {
    DeviceCtx *d = nullptr;
    PLK_TRY(device_ctx(device, &d));
    const bool c64 = dtype == PLK_C64;
    PLK_TRY(check_program(P, c64 ? 8 : 16));
    const Shape sh = shape(dtype, P.bwd);
    const int threads = std::max(32, 1 << (P.T - P.R));
    const int ntiles = 1 << (P.nq - P.T);
    // one resident wave: CTAs walk their tiles
    const int per_sm = std::min(sh.ctas * sh.threads / threads, 8);
    // a tile of fewer threads than a warp is worked on by several lanes alike
    const double share = (double)(1 << (P.T - P.R)) / threads;
    const int gx = std::max(1, std::min(ntiles, d->sm_count * per_sm / nsweep));
    // one device buffer: blobs, Jacobian terms, partial sums, Jacobian
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    std::vector<size_t> at;
    size_t up = 0;
    for (const TilePass &p : P.passes) {
        at.push_back(up);
        up += al(p.blob.size());
    }
    const size_t o_first = up, o_acc = o_first + al(sizeof(int) * (nslots + 1));
    const size_t o_coef = o_acc + al(sizeof(int) * P.jac.size()), o_end = o_coef + al(sizeof(double) * P.jac.size());
    if (P.bwd) up = o_end;
    const size_t o_part = up, b_part = P.bwd ? al(sizeof(double) * (size_t)nsweep * P.nacc * gx) : 0;
    const size_t o_jac = o_part + b_part, b_jac = P.bwd ? sizeof(double) * (size_t)nsweep * nslots : 0;
    std::vector<unsigned char> host(up, 0);
    for (size_t i = 0; i < P.passes.size(); i++)
        std::memcpy(host.data() + at[i], P.passes[i].blob.data(), P.passes[i].blob.size());
    if (P.bwd) { // terms by slot
        int *first = reinterpret_cast<int *>(host.data() + o_first), *ta = reinterpret_cast<int *>(host.data() + o_acc);
        double *tc = reinterpret_cast<double *>(host.data() + o_coef);
        for (const JacTerm &t : P.jac) first[t.slot + 1]++;
        for (int s = 0; s < nslots; s++) first[s + 1] += first[s];
        std::vector<int> next(first, first + nslots);
        for (const JacTerm &t : P.jac) {
            ta[next[t.slot]] = t.acc;
            tc[next[t.slot]++] = t.coef * share;
        }
    }
    PoolBuf buf(st);
    PLK_CUDA(cudaMallocFromPoolAsync(&buf.p, o_jac + b_jac + 256, d->pool, st));
    unsigned char *dev = buf.as<unsigned char>();
    PLK_CUDA(cudaMemcpyAsync(dev, host.data(), up, cudaMemcpyHostToDevice, st));
    Args a;
    std::memset((void *)&a, 0, sizeof(a));
    for (int y = 0; y < nsweep; y++) {
        a.lam_src[y] = lam_src[y];
        a.lam[y] = lam[y];
        a.hl[y] = P.bwd ? hl[y] : nullptr;
        if (words) {
            a.wx[y] = words[y].x;
            a.wz[y] = words[y].z;
            a.wq[y] = (uint8_t)(words[y].ny & 3);
        }
    }
    a.T = P.T;
    a.ntiles = ntiles;
    a.nacc_all = P.nacc;
    a.part = reinterpret_cast<double *>(dev + o_part);
    const dim3 grid(gx, nsweep);
    // index maps alone: amplitudes are moved bit for bit (split into 48 bits and joined
    // again they came out up to 2^-49 off)
    bool moves_only = !P.bwd;
    for (const TilePass &p : P.passes)
        moves_only = moves_only && reinterpret_cast<const TileHdr *>(p.blob.data())->nstages == 0;
    for (size_t i = 0; i < P.passes.size(); i++) {
        const TileHdr &h = *reinterpret_cast<const TileHdr *>(P.passes[i].blob.data());
        a.prog = dev + at[i];
        a.prog_bytes = h.bytes;
        a.nacc = h.nacc;
        a.in_df = moves_only ? 2 : i > 0;
        a.words = words && i == 0;
        a.out_df = moves_only ? 2 : i + 1 < P.passes.size();
        a.drop = words && i + 1 == P.passes.size(); // their states are scratch
        const size_t smem = smem_bytes(c64 ? 8 : 16, P.bwd, P.T, h.bytes, h.nacc, threads);
        if (c64) PLK_TRY(launch_c64(P.bwd, a, grid, threads, smem, st));
        else if (P.bwd) PLK_TRY(launch_c128_bwd(a, grid, threads, smem, st));
        else PLK_TRY(launch_c128_fwd(a, grid, threads, smem, st));
        for (int y = 0; y < nsweep; y++) a.lam_src[y] = lam[y];
    }
    if (P.bwd && nslots > 0) {
        double *dj = reinterpret_cast<double *>(dev + o_jac);
        k_tile_jac<<<dim3((nslots + 7) / 8, nsweep), 256, 0, st>>>(
            a.part, gx, P.nacc, reinterpret_cast<const int *>(dev + o_first), reinterpret_cast<const int *>(dev + o_acc),
            reinterpret_cast<const double *>(dev + o_coef), nslots, dj);
        PLK_CHECK_LAUNCH();
        PLK_CUDA(cudaMemcpyAsync(jac_host, dj, b_jac, cudaMemcpyDeviceToHost, st));
        PLK_CUDA(cudaStreamSynchronize(st));
    }
    return PLK_OK;
}

// an op that the per-op path would accept
static bool well_formed(plk_state s, const plk_op &op) {
    if (op.gate <= PLK_GATE_IDENTITY || op.gate >= PLK_GATE_MATRIX) return false;
    const int nw = plk_gate_num_wires(op.gate), np = plk_gate_num_params(op.gate);
    if (nw > 0 ? op.num_wires != nw : op.num_wires < 1) return false;
    if (op.num_params < np || (op.num_params > 0 && !op.params)) return false;
    return check_wires(s, op.wires, op.num_wires) == PLK_OK;
}

static bool has_generator(int gate, int nw) {
    GatePlan p;
    return plan_generator(gate, nw, p) == PLK_OK;
}

static bool usable(plk_state s) {
    return window_path_enabled() && (s->dtype == PLK_C64 || c128_use_df()) && s->nq >= kMaxRegBits && s->nq <= 32;
}

// The whole op list as passes; handled stays false when an op is not of this
// path (dense matrices) or not well formed (the per-op path reports it).
//
// From four ops on.  Lists of alternating RX and CNOT, us as passes / op by op:
// 4 ops 10 qubits 12 / 14 (complex64) and 13 / 15 (complex128), 20 qubits 12 / 17
// and 19 / 25, 26 qubits 187 / 476 and 653 / 948; 12 ops 18 / 38, 19 / 46, 22 / 50,
// 26 / 74, 416 / 1435, 1101 / 2851.  Three such ops are about even up to 20 qubits,
// and three that touch a quarter of the state each (CZ) move less than a pass does.
int apply_ops(plk_state s, const plk_op *ops, int nops, bool &handled) {
    handled = false;
    if (!usable(s) || nops < 4) return PLK_OK;
    Compiler c(s->nq, false, options(s->nq, s->dtype, false));
    Lowered L;
    for (int i = 0; i < nops; i++) {
        if (ops[i].gate == PLK_GATE_IDENTITY) continue;
        L.v.clear();
        if (!well_formed(s, ops[i]) || !lower_op(ops[i], s->nq, -1, L)) return PLK_OK;
        c.add(L.v);
    }
    TileProgram P;
    if (!c.compile(P)) return PLK_OK;
    handled = true;
    const void *src[1] = {s->data};
    void *dst[1] = {s->data};
    return run(P, s->dtype, s->device, s->stream, src, dst, nullptr, 1, 0, nullptr);
}

// The backward program of a tape; ok stays false when an op is not of this path.
static int compile_backward(plk_state lam, const plk_op *ops, int nops, const int64_t *tp, int ntp, TileProgram &P,
                            std::vector<SweptOp> &swept, bool &ok) {
    ok = false;
    swept.clear();
    int num_param_ops = 0;
    for (int i = 0; i < nops; i++)
        if (ops[i].num_params > 0) num_param_ops++;
    // the reference's backward walk: ops in reverse until every trainable
    // parameter is done (AdjointDiffKokkos.hpp:436-470)
    Compiler c(lam->nq, true, options(lam->nq, lam->dtype, true));
    Lowered L;
    long current_param_idx = num_param_ops - 1;
    int tp_it = ntp - 1;
    for (int i = nops - 1; i >= 0 && tp_it >= 0; i--) {
        const plk_op &op = ops[i];
        if (op.num_params > 1) return PLK_OK; // rejected by the reference; the per-op path reports it
        const bool trainable = op.num_params > 0 && current_param_idx == tp[tp_it];
        if (op.gate != PLK_GATE_IDENTITY) {
            L.v.clear();
            if (!well_formed(lam, op) || (trainable && !has_generator(op.gate, op.num_wires)) ||
                !lower_op(op, lam->nq, trainable ? tp_it : -1, L))
                return PLK_OK;
            invert(L.v);
            c.add(L.v);
            swept.push_back({op.gate, trainable});
        } else if (trainable) {
            return PLK_OK;
        }
        if (trainable) tp_it--;
        if (op.num_params > 0) current_param_idx--;
    }
    ok = c.compile(P) && !P.passes.empty();
    return PLK_OK;
}

// Backward sweeps of all observables; lam is the working copy of the forward
// state (overwritten).  plain: the tape is of this path, but cheaper op by op.
int adjoint(plk_state lam, plk_state *hls, int nobs, const plk_op *ops, int nops, const int64_t *tp, int ntp,
            double *jac, bool &handled, bool &plain) {
    handled = plain = false;
    if (!usable(lam) || ntp <= 0 || nobs < 1) return PLK_OK;
    TileProgram P;
    std::vector<SweptOp> swept;
    bool ok = false;
    PLK_TRY(compile_backward(lam, ops, nops, tp, ntp, P, swept, ok));
    if (!ok) return PLK_OK;
    plain = !tiles_pay(nobs, lam->dtype == PLK_C64, P, swept);
    if (plain) return PLK_OK;
    // several sweeps start from lambda: each works on its own copy
    const size_t bytes = lam->length * amp_bytes(lam->dtype);
    int group = std::min(nobs, kMaxSweeps);
    PoolBuf copies(lam->stream);
    if (nobs > 1) {
        const size_t most = (size_t)2 << 30;
        group = (int)std::min<size_t>(group, std::max<size_t>(1, most / bytes));
        if (pool_alloc(lam->device, &copies.p, bytes * group, lam->stream) != PLK_OK) {
            // no room for a copy of lambda: the op-at-a-time path needs none
            cudaGetLastError();
            set_error(std::string());
            return PLK_OK;
        }
    }
    handled = true;
    for (int o0 = 0; o0 < nobs; o0 += group) {
        const int n = std::min(group, nobs - o0);
        const void *src[kMaxSweeps];
        void *dst[kMaxSweeps], *h[kMaxSweeps];
        for (int y = 0; y < n; y++) {
            src[y] = lam->data;
            h[y] = hls[o0 + y]->data;
            dst[y] = nobs == 1 ? lam->data : copies.as<char>() + bytes * y;
        }
        PLK_TRY(run(P, lam->dtype, lam->device, lam->stream, src, dst, h, n, ntp, jac + (size_t)o0 * ntp));
    }
    if (nobs > 1) // lambda ends as the swept state, as with one observable
        PLK_CUDA(cudaMemcpyAsync(lam->data, copies.p, bytes, cudaMemcpyDeviceToDevice, lam->stream));
    return PLK_OK;
}

// Words whose tape is cheaper gate by gate: their states are formed here, so that
// the caller does not compile the tape once more to learn the same (22 qubits
// complex64, 100 DoubleExcitation, three PauliZ: 3.33 ms when it did, 2.94 so).
static int adjoint_word_states(plk_state lam, const std::vector<Word> &words, const plk_op *ops, int nops,
                               const int64_t *tp, int ntp, double *jac) {
    std::vector<plk_state> made; // the working copy of lambda, then H lambda of each word
    int rc = PLK_OK;
    for (size_t o = 0; o <= words.size() && rc == PLK_OK; o++) {
        plk_state s = nullptr;
        rc = plk_state_create(lam->nq, lam->dtype, lam->device, &s);
        if (rc != PLK_OK) break;
        made.push_back(s);
        rc = plk_state_set_stream(s, lam->stream);
        if (rc == PLK_OK) rc = plk_state_copy(s, lam);
        for (int b = 0; o > 0 && b < lam->nq && rc == PLK_OK; b++) {
            const Word &w = words[o - 1];
            const int gate = (w.x & w.z) >> b & 1 ? PLK_GATE_PAULIY : w.x >> b & 1 ? PLK_GATE_PAULIX : PLK_GATE_PAULIZ;
            const int64_t wire = lam->nq - 1 - b;
            if ((w.x | w.z) >> b & 1) rc = plk_apply_gate(s, gate, &wire, 1, 0, nullptr, 0);
        }
    }
    if (rc == PLK_OK) rc = adjoint_gates(made[0], made.data() + 1, (int)words.size(), ops, nops, tp, ntp, jac);
    const std::string err = rc == PLK_OK ? std::string() : last_error();
    for (plk_state s : made) plk_state_destroy(s);
    if (rc != PLK_OK) set_error(err);
    return rc;
}

// Observables that are one Pauli word each: H lambda is never stored, the first
// pass reads it as the permuted, signed lambda (which is not modified).
static int adjoint_words(plk_state lam, const std::vector<Word> &words, const plk_op *ops, int nops, const int64_t *tp,
                         int ntp, double *jac, bool &handled) {
    handled = false;
    const int nobs = (int)words.size();
    if (!usable(lam) || ntp <= 0 || nobs < 1) return PLK_OK;
    TileProgram P;
    std::vector<SweptOp> swept;
    bool ok = false;
    PLK_TRY(compile_backward(lam, ops, nops, tp, ntp, P, swept, ok));
    if (!ok) return PLK_OK;
    const bool gates = !tiles_pay(nobs, lam->dtype == PLK_C64, P, swept);
    DeviceCtx *d = nullptr;
    PLK_TRY(device_ctx(lam->device, &d));
    const size_t bytes = std::max<size_t>(256, lam->length * amp_bytes(lam->dtype));
    const int group =
        (int)std::min<size_t>(std::min(nobs, kMaxSweeps), std::max<size_t>(1, ((size_t)4 << 30) / (2 * bytes)));
    PoolBuf buf(lam->stream);
    if (gates) {
        PLK_TRY(adjoint_word_states(lam, words, ops, nops, tp, ntp, jac));
    } else if (cudaMallocFromPoolAsync(&buf.p, 2 * bytes * group, d->pool, lam->stream) != cudaSuccess) {
        cudaGetLastError();
        buf.p = nullptr;
        return PLK_OK; // the caller has ways that need less
    }
    handled = true;
    for (int o0 = 0; o0 < nobs && !gates; o0 += group) {
        const int n = std::min(group, nobs - o0);
        const void *src[kMaxSweeps];
        void *dst[kMaxSweeps], *h[kMaxSweeps];
        for (int y = 0; y < n; y++) {
            src[y] = lam->data;
            dst[y] = buf.as<char>() + 2 * bytes * y;
            h[y] = buf.as<char>() + 2 * bytes * y + bytes;
        }
        PLK_TRY(run(P, lam->dtype, lam->device, lam->stream, src, dst, h, n, ntp, jac + (size_t)o0 * ntp, &words[o0]));
    }
    for (int o = 0; o < nobs; o++) // the sweeps ran on the bare words
        for (int t = 0; t < ntp; t++) jac[(size_t)o * ntp + t] *= words[o].coeff;
    return PLK_OK;
}

} // namespace tile

int adjoint_checks(plk_state lambda, plk_state *hlambda, int32_t nobs, const plk_op *ops, int32_t nops,
                   const int64_t *trainable, int32_t ntp, double *jac);

} // namespace plk

using namespace plk;

extern "C" {

PLK_API int plk_adjoint_jacobian_pauli(plk_state lambda, int32_t num_obs, const double *coeffs, const int64_t *offsets,
                                       const int64_t *wires, const char *paulis, const plk_op *ops, int32_t num_ops,
                                       const int64_t *trainable, int32_t num_trainable, double *jac) {
    PLK_TRY(adjoint_checks(lambda, nullptr, 0, ops, num_ops, trainable, num_trainable, jac));
    if (num_obs < 1 || !coeffs || !offsets) PLK_FAIL(PLK_ERR_INVALID_ARG, "bad Pauli-word arguments");
    PLK_CUDA(cudaSetDevice(lambda->device));
    if (lambda->nq > 32) PLK_FAIL(PLK_ERR_UNSUPPORTED, "this state's sweeps do not start from Pauli words");
    std::vector<tile::Word> words;
    for (int o = 0; o < num_obs; o++) {
        tile::Word w{0, 0, 0, coeffs[o]};
        if (offsets[o + 1] < offsets[o]) PLK_FAIL(PLK_ERR_INVALID_ARG, "Pauli-word offsets must be non-decreasing");
        for (int64_t j = offsets[o]; j < offsets[o + 1]; j++) {
            if (!wires || !paulis) PLK_FAIL(PLK_ERR_INVALID_ARG, "bad Pauli-word arguments");
            if (wires[j] < 0 || wires[j] >= lambda->nq) PLK_FAIL(PLK_ERR_INVALID_ARG, "Pauli word wire out of range");
            const uint32_t bit = 1u << (lambda->nq - 1 - wires[j]);
            if ((w.x | w.z) & bit) PLK_FAIL(PLK_ERR_INVALID_ARG, "repeated wire in a Pauli word");
            switch (paulis[j]) {
            case 'I': break;
            case 'X': w.x |= bit; break;
            case 'Y': w.x |= bit; w.z |= bit; w.ny++; break;
            case 'Z': w.z |= bit; break;
            default: PLK_FAIL(PLK_ERR_INVALID_ARG, std::string("bad Pauli letter ") + paulis[j]);
            }
        }
        words.push_back(w);
    }
    bool handled = false;
    PLK_TRY(tile::adjoint_words(lambda, words, ops, num_ops, trainable, num_trainable, jac, handled));
    if (!handled) PLK_FAIL(PLK_ERR_UNSUPPORTED, "this tape's sweep does not start from Pauli words");
    return PLK_OK;
}

} // extern "C"
