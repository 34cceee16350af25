// pauli_tile.cu — expectation value and application of Pauli sums on tiles
// (MeasuresKokkos / ObservablesKokkos.hpp:296-402 Hamiltonians of Pauli terms;
// the reference materialises each term).
//
// A CTA of 256 threads loads a tile of 2^12 amplitudes (complex64 32 KiB;
// complex128 64 KiB as double-float pairs), each thread keeps its 16 amplitudes
// (the top four tile bits) in registers and reads partners m ^ x from shared
// memory: lanes differ in the low tile bits, so a read touches consecutive slots
// permuted by an exclusive or, free of bank conflicts.  Smaller states use one
// tile of all their bits; the threads that are left over take other words.
//
// Expectation value: each pair (m, m ^ x) is visited once, eight pairs per
// thread and word; when x has none of the register bits, the thread with bit p
// of x clear takes its lower eight amplitudes and its partner thread the upper
// eight.  Re or Im of conj(a) b accumulates with the word's sign, then takes the
// coefficient once per thread: complex64 forms eight products per lane in FP32,
// then double-float; complex128 is double-float throughout, packed two lanes per
// instruction (the one-pass kernel formed its products on the FP64 pipe, whose
// rate bounded it).  100 words, one GB300: 26-qubit complex128 expectation value
// 19.3 -> 5.6 ms, 25-qubit complex128 application 15.8 -> 5.6 ms, 26-qubit
// complex64 10.9 -> 3.3 ms and 8.2 -> 3.7 ms; now bound by the FP32 pipe
// (complex128) and by shared-memory reads (complex64).  Words that share x form their products once and pick their
// signed sums from a Walsh transform over the pairs.
#include <algorithm>
#include <cstring>

#include "pauli_tile.cuh"
#include "reduce.cuh"
#include "tile_kernels.cuh"

namespace plk {

using tile::AmpC128;
using tile::AmpC64;
using tile::f2x_hi;
using tile::f2x_lo;
using tile::ins0;

namespace {

constexpr int kPT = 12, kPR = 4, kPA = 1 << kPR; // tile bits, register bits

enum ItemKind : uint32_t { PI_DIAG = 0, PI_RE = 1, PI_IM = 2, PI_MANY = 3 };
struct alignas(16) Item {
    uint32_t x;     // byte offset in the tile (exclusive or)
    uint32_t kind;
    uint32_t z;     // sign bits of the state index
    uint32_t zr;    // those on register bits
    int32_t p;      // register bit in x, or -1 - (thread bit in x)
    uint32_t first, count; // PI_DIAG, PI_MANY: terms
    uint32_t xs;    // x as state bits
    float ch, cl;   // coefficient (real part, or imaginary part of c i^ny)
    uint32_t pad[2];
};
struct alignas(16) Term {
    uint32_t z, zr;
    uint32_t odd; // parity of x & z: the imaginary product enters
    float ch, cl;
    uint32_t pad[3];
};

struct PauliArgs {
    const void *in;
    void *out;
    const Item *items;
    const Term *terms;
    int nitems;
    int T, ntiles, tiles_x; // tiles_x CTAs walk the tiles, gridDim.x / tiles_x share the items
    int accumulate;
    uint8_t gpos[16];       // state bit of tile bit k (ascending)
};

constexpr f2x kSigns = 0x8000000080000000ull;

template <class A> __device__ __forceinline__ typename A::V flip(typename A::V v, f2x m);
template <> __device__ __forceinline__ f2x flip<AmpC64>(f2x v, f2x m) { return v ^ m; }
template <> __device__ __forceinline__ AmpC128::V flip<AmpC128>(AmpC128::V v, f2x m) { return {v.h ^ m, v.l ^ m}; }
__device__ __forceinline__ f2x choose(bool c, f2x a, f2x b) { return c ? a : b; }
__device__ __forceinline__ AmpC128::V choose(bool c, AmpC128::V a, AmpC128::V b) { return {c ? a.h : b.h, c ? a.l : b.l}; }

// state offset of this thread's amplitudes, relative to the tile
__device__ __forceinline__ uint32_t thread_bits(const PauliArgs &a, int tl) {
    uint32_t g = 0;
    for (int i = 0; i < a.T - kPR; i++)
        if (tl >> i & 1) g |= 1u << a.gpos[i];
    return g;
}
__device__ __forceinline__ uint32_t tile_base(const PauliArgs &a, int tile) {
    uint32_t base = (uint32_t)tile;
    for (int k = 0; k < a.T; k++) {
        const uint32_t lo = base & ((1u << a.gpos[k]) - 1u);
        base = ((base ^ lo) << 1) | lo;
    }
    return base;
}

// Re (IM: Im) of conj(a) b over eight pairs, signed by the parity of j & zr;
// tx: byte offset of this thread's partners, js: bytes between register indices
template <class A, int B, bool IM>
__device__ __forceinline__ DF pairs(const typename A::V (&v)[kPA], const unsigned char *L, uint32_t tx, uint32_t js,
                                    uint32_t zr, bool half) {
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = B < 4 ? ins0(i, B < 4 ? B : 0) : i; // B = 4: this thread's lower or upper eight
        typename A::V x = v[j];
        if (B == 4) x = choose(half, v[(i | 8) & 15], v[i]);
        const typename A::V y = A::ld(L + (tx ^ (uint32_t)j * js));
        const f2x m = (__popc(j & zr) & 1) ? kSigns : 0ull;
        x = flip<A>(x, m);
        if constexpr (A::kBytes == 8) {
            sh = f2x_fma(x, IM ? f2x_swap(y) : y, sh);
        } else {
            tile::pdf_mac(x.h, x.h ^ kSigns, x.l, IM ? f2x_swap(y.h) : y.h, IM ? f2x_swap(y.l) : y.l, sh, sl);
        }
    }
    // lanes (re re, im im), or (re im, im re)
    DF r = {f2x_lo(sh), f2x_lo(sl)};
    if (IM) df_add(-f2x_hi(sh), -f2x_hi(sl), r.hi, r.lo);
    else df_add(f2x_hi(sh), f2x_hi(sl), r.hi, r.lo);
    return r;
}

__device__ __forceinline__ void products(f2x a, f2x b, DF &re, DF &im) {
    const float ar = f2x_lo(a), ai = f2x_hi(a), br = f2x_lo(b), bi = f2x_hi(b);
    re = {fmaf(ar, br, ai * bi), 0.0f};
    im = {fmaf(ar, bi, -ai * br), 0.0f};
}
__device__ __forceinline__ void products(const AmpC128::V &a, const AmpC128::V &b, DF &re, DF &im) {
    const DF ar = {f2x_lo(a.h), f2x_lo(a.l)}, ai = {f2x_hi(a.h), f2x_hi(a.l)};
    const DF br = {f2x_lo(b.h), f2x_lo(b.l)}, bi = {f2x_hi(b.h), f2x_hi(b.l)};
    df_first(ar.hi, ar.lo, br.hi, br.lo, re.hi, re.lo);
    df_mac(ai.hi, ai.lo, bi.hi, bi.lo, re.hi, re.lo);
    df_first(ar.hi, ar.lo, bi.hi, bi.lo, im.hi, im.lo);
    df_mac(-ai.hi, -ai.lo, br.hi, br.lo, im.hi, im.lo);
}

// w <- its Walsh transform (N = 2^K double-floats)
template <int K> __device__ __forceinline__ void walsh(DF (&w)[1 << K]) {
#pragma unroll
    for (int b = 0; b < K; b++)
#pragma unroll
        for (int p = 0; p < 1 << (K - 1); p++) {
            const int i = ins0(p, b), k = i | 1 << b;
            const DF s = tile::plus(w[i], w[k]);
            DF d = w[i];
            df_add(-w[k].hi, -w[k].lo, d.hi, d.lo);
            w[i] = s;
            w[k] = d;
        }
}
template <int N> __device__ __forceinline__ DF pick_of(const DF (&w)[N], uint32_t k) {
    DF r = w[0];
#pragma unroll
    for (int i = 1; i < N; i++) r = tile::pick(k == (uint32_t)i, w[i], r);
    return r;
}

template <class A> struct Ctas;
template <> struct Ctas<AmpC64> {
    static constexpr int expval = 3, apply = 3;
};
template <> struct Ctas<AmpC128> {
    static constexpr int expval = 2, apply = 2;
};

template <class A>
__device__ __forceinline__ void load(const PauliArgs &a, uint32_t g, const uint32_t (&gr)[kPR], unsigned char *L, int tl,
                                     uint32_t js, bool store, typename A::V (&v)[kPA]) {
#pragma unroll
    for (int j = 0; j < kPA; j++) {
        const uint32_t i = g | ((j & 1) ? gr[0] : 0u) | ((j & 2) ? gr[1] : 0u) | ((j & 4) ? gr[2] : 0u) |
                           ((j & 8) ? gr[3] : 0u);
        v[j] = tile::load_amp(a.in, i, 0, typename A::V{});
        if (store) A::st(L + (uint32_t)tl * A::kBytes + (uint32_t)j * js, v[j]);
    }
}

template <class A>
__global__ void __launch_bounds__(kThreads, Ctas<A>::expval)
    k_pauli_expval_tile(const __grid_constant__ PauliArgs a, double *partials, double *result, unsigned *counter) {
    using V = typename A::V;
    extern __shared__ __align__(16) unsigned char pauli_smem[];
    const int per = 1 << (a.T - kPR);            // threads of the tile
    const int tl = threadIdx.x & (per - 1), grp = threadIdx.x / per, groups = kThreads / per;
    const uint32_t js = (uint32_t)A::kBytes << (a.T - kPR);
    const int cx = blockIdx.x % a.tiles_x, cy = blockIdx.x / a.tiles_x, ny = gridDim.x / a.tiles_x;
    const uint32_t gt = thread_bits(a, tl);
    uint32_t gr[kPR];
#pragma unroll
    for (int i = 0; i < kPR; i++) gr[i] = 1u << a.gpos[a.T - kPR + i];
    DAcc total;
    for (int tile = cx; tile < a.ntiles; tile += a.tiles_x) {
        const uint32_t g = tile_base(a, tile) | gt;
        V v[kPA];
        load<A>(a, g, gr, pauli_smem, tl, js, grp == 0, v);
        __syncthreads();
        for (int k = cy * groups + grp; k < a.nitems; k += ny * groups) {
            const Item it = a.items[k];
            const uint32_t tx = (uint32_t)tl * A::kBytes ^ it.x;
            if (it.kind == PI_RE || it.kind == PI_IM) {
                DF r;
                bool neg = __popc(g & it.z) & 1;
                if (it.p >= 0) {
#define PLK_PAIRS(B) r = it.kind == PI_RE ? pairs<A, B, false>(v, pauli_smem, tx, js, it.zr, false)                     \
                                          : pairs<A, B, true>(v, pauli_smem, tx, js, it.zr, false)
                    switch (it.p) {
                    case 0: PLK_PAIRS(0); break;
                    case 1: PLK_PAIRS(1); break;
                    case 2: PLK_PAIRS(2); break;
                    default: PLK_PAIRS(3); break;
                    }
#undef PLK_PAIRS
                } else {
                    const bool half = tl >> (-1 - it.p) & 1;
                    if (half) neg = neg != (bool)(it.zr >> 3 & 1);
                    const uint32_t th = tx ^ (half ? 8u * js : 0u);
                    r = it.kind == PI_RE ? pairs<A, 4, false>(v, pauli_smem, th, js, it.zr & 7u, half)
                                         : pairs<A, 4, true>(v, pauli_smem, th, js, it.zr & 7u, half);
                }
                const float ch = neg ? -it.ch : it.ch, cl = neg ? -it.cl : it.cl;
                df_mac(ch, cl, r.hi, r.lo, total.h, total.l);
            } else if (it.kind == PI_DIAG) {
                DF w[kPA];
#pragma unroll
                for (int j = 0; j < kPA; j++) {
                    DF im;
                    products(v[j], v[j], w[j], im);
                }
                walsh<kPR>(w);
                for (uint32_t t = it.first; t < it.first + it.count; t++) {
                    const Term tt = a.terms[t];
                    const bool neg = __popc(g & tt.z) & 1;
                    const DF r = pick_of<kPA>(w, tt.zr);
                    df_mac(neg ? -tt.ch : tt.ch, neg ? -tt.cl : tt.cl, r.hi, r.lo, total.h, total.l);
                }
            } else {
                // pair i: j = i with a clear bit p inserted (p in registers), or
                // this thread's lower or upper eight
                DF re[8], im[8];
                const bool inreg = it.p >= 0;
                const bool half = !inreg && (tl >> (-1 - it.p) & 1);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    V x = choose(half, v[i | 8], v[i]);
                    int j = half ? i | 8 : i;
                    if (inreg) {
                        j = ins0(i, it.p);
#pragma unroll
                        for (int q = 0; q < 4; q++) x = choose(it.p == q, v[ins0(i, q)], x);
                    }
                    products(x, A::ld(pauli_smem + (tx ^ (uint32_t)j * js)), re[i], im[i]);
                }
                walsh<3>(re);
                walsh<3>(im);
                for (uint32_t t = it.first; t < it.first + it.count; t++) {
                    const Term tt = a.terms[t];
                    bool neg = __popc(g & tt.z) & 1;
                    uint32_t w = tt.zr & 7u;
                    if (inreg) w = (tt.zr & ((1u << it.p) - 1u)) | ((tt.zr >> (it.p + 1)) << it.p);
                    else if (half) neg = neg != (bool)(tt.zr >> 3 & 1);
                    const DF r = tt.odd ? pick_of<8>(im, w) : pick_of<8>(re, w);
                    df_mac(neg ? -tt.ch : tt.ch, neg ? -tt.cl : tt.cl, r.hi, r.lo, total.h, total.l);
                }
            }
        }
        __syncthreads();
    }
    double acc[1] = {total.value()};
    block_reduce_finish<1>(acc, partials, result, counter);
}

// out (+)= sum over items of c i^ny (-1)^popcount(src & z) in[src], src = m ^ x
template <class A>
__global__ void __launch_bounds__(kThreads, Ctas<A>::apply) k_pauli_apply_tile(const __grid_constant__ PauliArgs a) {
    using V = typename A::V;
    extern __shared__ __align__(16) unsigned char pauli_smem[];
    const int per = 1 << (a.T - kPR);
    const int tl = threadIdx.x & (per - 1);
    const uint32_t js = (uint32_t)A::kBytes << (a.T - kPR);
    const uint32_t gt = thread_bits(a, tl);
    uint32_t gr[kPR];
#pragma unroll
    for (int i = 0; i < kPR; i++) gr[i] = 1u << a.gpos[a.T - kPR + i];
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const uint32_t g = tile_base(a, tile) | gt;
        auto at = [&](int j) {
            return g | ((j & 1) ? gr[0] : 0u) | ((j & 2) ? gr[1] : 0u) | ((j & 4) ? gr[2] : 0u) | ((j & 8) ? gr[3] : 0u);
        };
        V s[kPA];
        load<A>(a, g, gr, pauli_smem, tl, js, true, s);
#pragma unroll
        for (int j = 0; j < kPA; j++) s[j] = a.accumulate ? tile::load_amp(a.out, at(j), 0, V{}) : V{};
        __syncthreads();
        for (int k = 0; k < a.nitems; k++) {
            const Item it = a.items[k];
            const uint32_t tx = (uint32_t)tl * A::kBytes ^ it.x;
            const bool neg = __popc((g ^ it.xs) & it.z) & 1;
            const bool im = it.kind == PI_IM;
            // lanes of the coefficient: (c, c), or (-c, c) on the swapped amplitude
            const float c = neg ? -it.ch : it.ch, cl = neg ? -it.cl : it.cl;
            const f2x ch2 = f2x_pack(im ? -c : c, c), cl2 = f2x_pack(im ? -cl : cl, cl);
#pragma unroll
            for (int j = 0; j < kPA; j++) {
                V y = A::ld(pauli_smem + (tx ^ (uint32_t)j * js));
                const f2x m = (__popc(j & it.zr) & 1) ? kSigns : 0ull;
                if constexpr (A::kBytes == 8) {
                    if (im) y = f2x_swap(y);
                    s[j] = f2x_fma(ch2 ^ m, y, s[j]);
                } else {
                    if (im) y = {f2x_swap(y.h), f2x_swap(y.l)};
                    const f2x h = ch2 ^ m;
                    tile::pdf_mac(h, h ^ kSigns, cl2 ^ m, y.h, y.l, s[j].h, s[j].l);
                }
            }
        }
        __syncthreads(); // partners read before the next tile is loaded
#pragma unroll
        for (int j = 0; j < kPA; j++) tile::store_amp(a.out, at(j), 0, s[j]);
    }
}

// --------------------------------------------------------------- host side --
struct Pass {
    uint32_t bits = 0;       // state bits of the tile
    std::vector<int> groups; // indices of the groups inside
};

int popc(uint64_t x) { return __builtin_popcountll(x); }

// Tiles that cover the groups' X patterns: each pass starts from the widest
// pattern left, adds patterns that need the fewest more bits, and takes every
// group that lies inside.
void choose_passes(int nq, int T, int low, const std::vector<PauliGroup> &groups, std::vector<Pass> &passes,
                   std::vector<PauliGroup> &rest) {
    const uint64_t lowmask = (1ull << low) - 1;
    std::vector<char> done(groups.size(), 0);
    std::vector<int> order(groups.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return popc(groups[a].x & ~lowmask) > popc(groups[b].x & ~lowmask);
    });
    for (int seed : order) {
        if (done[seed]) continue;
        uint64_t bits = lowmask;
        Pass p;
        if (T < nq && popc(bits | groups[seed].x) > T) {
            done[seed] = 1;
            rest.push_back(groups[seed]);
            continue;
        }
        bits |= groups[seed].x;
        for (;;) {
            int best = -1, cost = 0;
            for (int i : order) {
                if (done[i] || (groups[i].x & ~bits) == 0) continue;
                const int c = popc(bits | groups[i].x);
                if (c <= T && (best < 0 || c < cost)) {
                    best = i;
                    cost = c;
                }
            }
            if (best < 0) break;
            bits |= groups[best].x;
        }
        for (int b = 0; b < nq && popc(bits) < T; b++) bits |= 1ull << b;
        p.bits = (uint32_t)bits;
        for (size_t i = 0; i < groups.size(); i++)
            if (!done[i] && (groups[i].x & ~bits) == 0) {
                done[i] = 1;
                p.groups.push_back((int)i);
            }
        // one group alone: a plain pass reads the state as often
        if (p.groups.size() == 1 && T < nq) rest.push_back(groups[p.groups[0]]);
        else passes.push_back(std::move(p));
    }
}

struct Plan {
    std::vector<Pass> passes;
    std::vector<Item> items;
    std::vector<Term> terms;
    std::vector<int> item0; // per pass (and one past)
    std::vector<PauliArgs> args;
};

// singles: every term its own item (application); else words that share x share an item
void make_plan(int nq, int dtype, const std::vector<PauliGroup> &groups, const std::vector<PauliTerm> &terms,
               bool singles, Plan &pl, std::vector<PauliGroup> &rest) {
    const int T = std::min(kPT, nq), amp = dtype == PLK_C64 ? 8 : 16;
    const int low = std::min(dtype == PLK_C64 ? 3 : 2, T);
    choose_passes(nq, T, low, groups, pl.passes, rest);
    for (const Pass &p : pl.passes) {
        PauliArgs a;
        std::memset((void *)&a, 0, sizeof(a));
        a.T = T;
        a.ntiles = 1 << (nq - T);
        int pos[32], n = 0;
        for (int b = 0; b < nq; b++)
            if (p.bits >> b & 1) {
                pos[b] = n;
                a.gpos[n++] = (uint8_t)b;
            }
        pl.args.push_back(a);
        pl.item0.push_back((int)pl.items.size());
        auto local = [&](uint64_t m) {
            uint32_t r = 0;
            for (; m; m &= m - 1) {
                const int b = __builtin_ctzll(m);
                if (p.bits >> b & 1) r |= 1u << pos[b];
            }
            return r;
        };
        for (int gi : p.groups) {
            const PauliGroup &g = groups[gi];
            Item it;
            std::memset(&it, 0, sizeof(it));
            const uint32_t xl = local(g.x);
            it.x = xl * amp;
            it.xs = (uint32_t)g.x;
            const uint32_t xr = xl >> (T - kPR);
            it.p = xr ? 31 - __builtin_clz(xr) : (xl ? -1 - (31 - __builtin_clz(xl)) : 0);
            auto single = [&](const PauliTerm &t, float scale) {
                const bool odd = popc(g.x & t.z) & 1;
                // c i^ny is real for an even number of Y, imaginary for an odd one
                it.kind = odd ? PI_IM : PI_RE;
                it.z = (uint32_t)t.z;
                it.zr = local(t.z) >> (T - kPR);
                it.ch = scale * (odd ? t.cih : t.crh);
                it.cl = scale * (odd ? t.cil : t.crl);
                pl.items.push_back(it);
            };
            if (singles) {
                for (int k = 0; k < g.count; k++) single(terms[g.first + k], 1.0f);
            } else if (g.count == 1 && g.x) {
                single(terms[g.first], 2.0f); // a pair counts twice
            } else {
                it.kind = g.x ? PI_MANY : PI_DIAG;
                it.first = (uint32_t)pl.terms.size();
                it.count = (uint32_t)g.count;
                for (int k = 0; k < g.count; k++) {
                    const PauliTerm &t = terms[g.first + k];
                    Term d;
                    std::memset(&d, 0, sizeof(d));
                    d.z = (uint32_t)t.z;
                    d.zr = local(t.z) >> (T - kPR);
                    d.odd = popc(g.x & t.z) & 1;
                    const float scale = g.x ? 2.0f : 1.0f;
                    d.ch = scale * (d.odd ? t.cih : t.crh);
                    d.cl = scale * (d.odd ? t.cil : t.crl);
                    pl.terms.push_back(d);
                }
                pl.items.push_back(it);
            }
        }
    }
    pl.item0.push_back((int)pl.items.size());
}

// items and terms on the device, in one block of the pool
int upload(const Plan &pl, int device, cudaStream_t st, PoolBuf &buf, const Item *&items, const Term *&terms) {
    DeviceCtx *d = nullptr;
    PLK_TRY(device_ctx(device, &d));
    const size_t bi = sizeof(Item) * pl.items.size(), bt = sizeof(Term) * pl.terms.size();
    std::vector<unsigned char> host(bi + bt + 16);
    if (bi) std::memcpy(host.data(), pl.items.data(), bi);
    if (bt) std::memcpy(host.data() + bi, pl.terms.data(), bt);
    PLK_CUDA(cudaMallocFromPoolAsync(&buf.p, host.size(), d->pool, st));
    PLK_CUDA(cudaMemcpyAsync(buf.p, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    items = buf.as<const Item>();
    terms = reinterpret_cast<const Term *>(buf.as<char>() + bi);
    return PLK_OK;
}

size_t smem_of(int dtype, int T) { return (size_t)(dtype == PLK_C64 ? 8 : 16) << T; }

template <class K> int opt_in(K kernel, size_t bytes) {
    if (bytes > 48 * 1024) PLK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return PLK_OK;
}

} // namespace

int pauli_tile_expval(plk_state s, const std::vector<PauliGroup> &groups, const std::vector<PauliTerm> &terms,
                      std::vector<PauliGroup> &rest, double &total) {
    total = 0.0;
    if (s->nq < kPR || s->nq > 32 || groups.size() < 2) {
        rest = groups;
        return PLK_OK;
    }
    Plan pl;
    make_plan(s->nq, s->dtype, groups, terms, false, pl, rest);
    if (pl.passes.empty()) return PLK_OK;
    PoolBuf buf(s->stream);
    const Item *items = nullptr;
    const Term *dterms = nullptr;
    PLK_TRY(upload(pl, s->device, s->stream, buf, items, dterms));
    const bool c64 = s->dtype == PLK_C64;
    const int T = pl.args[0].T;
    const size_t smem = smem_of(s->dtype, T);
    PLK_TRY(c64 ? opt_in(k_pauli_expval_tile<AmpC64>, smem) : opt_in(k_pauli_expval_tile<AmpC128>, smem));
    const int cap = device_sm_count(s->device) * (c64 ? Ctas<AmpC64>::expval : Ctas<AmpC128>::expval);
    const int groups_in_cta = kThreads >> (T - kPR);
    auto &w = s->ws;
    std::vector<double> vals(pl.passes.size());
    for (size_t i = 0; i < pl.passes.size(); i++) {
        PauliArgs a = pl.args[i];
        a.in = s->data;
        a.items = items + pl.item0[i];
        a.terms = dterms;
        a.nitems = pl.item0[i + 1] - pl.item0[i];
        a.tiles_x = std::min(a.ntiles, cap);
        // few tiles: CTAs share the words of a tile
        const int share = std::max(1, std::min(cap / a.tiles_x, (a.nitems + groups_in_cta - 1) / groups_in_cta));
        const int grid = a.tiles_x * share;
        double *res = w.d_result + (i % kMaxRedValues);
        if (c64) k_pauli_expval_tile<AmpC64><<<grid, kThreads, smem, s->stream>>>(a, w.d_partials, res, w.d_counter);
        else k_pauli_expval_tile<AmpC128><<<grid, kThreads, smem, s->stream>>>(a, w.d_partials, res, w.d_counter);
        PLK_CHECK_LAUNCH();
        if (i % kMaxRedValues == kMaxRedValues - 1 || i + 1 == pl.passes.size()) {
            const int nv = (int)(i % kMaxRedValues) + 1;
            PLK_TRY(fetch_results(s, nv, vals.data() + (i + 1 - nv)));
        }
    }
    for (double v : vals) total += v; // pass order
    return PLK_OK;
}

int pauli_tile_apply(plk_state out, plk_state in, const std::vector<PauliGroup> &groups,
                     const std::vector<PauliTerm> &terms, std::vector<PauliGroup> &rest, bool &accumulate) {
    // a tile pass reads the state and updates the output; a plain pass gathers
    // 32 patterns from the second-level cache or memory
    if (out->nq < kPT || out->nq > 32 || groups.size() < 2) {
        rest = groups;
        return PLK_OK;
    }
    Plan pl;
    make_plan(out->nq, out->dtype, groups, terms, true, pl, rest);
    if (pl.passes.empty()) return PLK_OK;
    cudaStream_t st = out->stream;
    PoolBuf buf(st);
    const Item *items = nullptr;
    const Term *dterms = nullptr;
    PLK_TRY(upload(pl, out->device, st, buf, items, dterms));
    const bool c64 = out->dtype == PLK_C64;
    const size_t smem = smem_of(out->dtype, pl.args[0].T);
    PLK_TRY(c64 ? opt_in(k_pauli_apply_tile<AmpC64>, smem) : opt_in(k_pauli_apply_tile<AmpC128>, smem));
    const int cap = device_sm_count(out->device) * (c64 ? Ctas<AmpC64>::apply : Ctas<AmpC128>::apply);
    for (size_t i = 0; i < pl.passes.size(); i++) {
        PauliArgs a = pl.args[i];
        a.in = in->data;
        a.out = out->data;
        a.items = items + pl.item0[i];
        a.terms = dterms;
        a.nitems = pl.item0[i + 1] - pl.item0[i];
        a.accumulate = accumulate;
        const int grid = std::min(a.ntiles, cap);
        if (c64) k_pauli_apply_tile<AmpC64><<<grid, kThreads, smem, st>>>(a);
        else k_pauli_apply_tile<AmpC128><<<grid, kThreads, smem, st>>>(a);
        PLK_CHECK_LAUNCH();
        accumulate = true;
    }
    return PLK_OK;
}

} // namespace plk
