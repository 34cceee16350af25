// pauli_tile.cu — expectation value and application of Pauli sums on tiles
// (MeasuresKokkos / ObservablesKokkos.hpp:296-402 Hamiltonians of Pauli terms;
// the reference materialises each term).
//
// A CTA of 256 threads loads a tile of 2^12 amplitudes into shared memory
// (complex64 32 KiB; complex128 64 KiB as double-float pairs).  A thread owns the
// 16 amplitudes that differ in four tile bits, the register bits, and reads
// partners m ^ x from shared memory: lanes differ in the other tile bits, so a
// read touches consecutive slots permuted by an exclusive or, free of bank
// conflicts.  Smaller states use one tile of all their bits; the threads that are
// left over take other words.
//
// Application: the thread's sums s_j += +-c in[m ^ x] stay in registers.  The
// sign is the product of a thread's part, which goes into the coefficient, and of
// the register bits' part, one three-input operation on the sign bit per index:
// complex64 flips the coefficient, complex128 forms the sum with fma(p, +-1, s),
// which costs no more than the addition.  Words with an odd number of Y carry a
// factor i: they come last, and s is turned by -i once for all of them.  Two words
// at a time: the second one's sum is written where the first found s, so that the
// loop needs no register moves.
//
// Expectation value: each pair (m, m ^ x) is visited once, eight pairs per thread
// and word; when x has none of the register bits, the thread with bit p of x clear
// takes its lower eight amplitudes and its partner thread the upper eight.
// Re conj(a) b accumulates with the word's sign, a turned by i for the words with
// an odd number of Y, then takes the coefficient once per thread: complex64 forms
// eight products per lane in FP32, then double-float; complex128 is double-float
// throughout.
//
// Words that share x and the factor, from a certain number on, form their
// coefficient per amplitude first: signed sums by register bits, then a Walsh
// transform (double-float).
//
// 100 random words of weight 1-4, one GB300, one pass over the state per X pattern
// (with products on the FP64 pipe) -> tiles with a sign formed per amplitude and
// word -> now: 26-qubit complex128 expectation value 19.1 -> 5.4 -> 5.05 ms;
// 24-qubit kernels, sum of the passes, second and third: complex128 application
// 2.90 -> 1.82 ms and expectation value 1.39 -> 1.29, complex64 0.88 -> 0.64 and
// 0.80 -> 0.67.  Bound by the FP32 pipe (complex128, 55-60 % of its cycles in the
// larger passes) and by integer operations and shared-memory reads (complex64).
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
constexpr int kPer = 1 << (kPT - kPR);           // slots between register indices, whatever T is

// From how many words with the same x and factor on the coefficients are formed
// per amplitude.  24 qubits, ten patterns of n words, us through a transform / word
// by word: application complex64 n = 6 465 / 406, 8 508 / 501, 10 540 / 593,
// complex128 3 743 / 663, 4 756 / 821; expectation value complex64 5 389 / 357,
// 6 384 / 407, complex128 2 423 / 350, 3 437 / 463.
constexpr int kManyApplyC64 = 9, kManyApplyC128 = 4, kManyExpvalC64 = 6, kManyExpvalC128 = 3;

struct alignas(16) Item {
    uint32_t w;   // bits 0-15 x as a byte offset in the tile (exclusive or), 16-19 sign bits on register
                  // bits, 20 factor i, 21 several words, 24-27 pairing bit of x
    uint32_t z;   // sign bits of the state index; several words: where their nine offsets are
    float ch, cl; // coefficient (real part, or imaginary part of c i^ny)
};
constexpr uint32_t kFactorI = 1u << 20, kMany = 1u << 21;
constexpr int kPairShift = 24, kNoPair = 15; // pairing bit: a register bit 0-3, 4 + a thread bit, none (x = 0)
struct alignas(16) Term {
    uint32_t z;
    uint32_t top; // the sign flips in the upper half of the register indices
    float ch, cl;
};

struct PauliArgs {
    const void *in;
    void *out;
    const Item *items;
    const Term *terms;
    const uint32_t *offs;
    int nitems, nreal; // the first nreal without a factor i
    int T, ntiles, tiles_x; // tiles_x CTAs walk the tiles, gridDim.x / tiles_x share the items
    int accumulate;
    int sum_df; // complex128: `out` holds double-float pairs on exit; what is accumulated to always does
    uint8_t gpos[kPT];      // state bits of the tile, ascending
    uint8_t tpos[kPT];      // those of the thread bits
    uint8_t rpos[kPR];      // and of the register bits
};

constexpr f2x kSigns = 0x8000000080000000ull;

__device__ __forceinline__ f2x choose(bool c, f2x a, f2x b) { return c ? a : b; }
__device__ __forceinline__ AmpC128::V choose(bool c, const AmpC128::V &a, const AmpC128::V &b) {
    return {c ? a.h : b.h, c ? a.l : b.l};
}

// state offset of this thread's amplitudes, relative to the tile
__device__ __forceinline__ uint32_t thread_bits(const PauliArgs &a, int tl) {
    uint32_t g = 0;
    for (int i = 0; i < a.T - kPR; i++)
        if (tl >> i & 1) g |= 1u << a.tpos[i];
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
__device__ __forceinline__ uint32_t at(uint32_t g, const uint32_t (&gr)[kPR], int j) {
    return g | ((j & 1) ? gr[0] : 0u) | ((j & 2) ? gr[1] : 0u) | ((j & 4) ? gr[2] : 0u) | ((j & 8) ? gr[3] : 0u);
}
template <class A> __device__ __forceinline__ uint32_t slot(int j) { return (uint32_t)(j * kPer * A::kBytes); }

// this thread's amplitudes of the tile, into shared memory if `store`
template <class A>
__device__ __forceinline__ void load(const PauliArgs &a, uint32_t g, const uint32_t (&gr)[kPR], unsigned char *own,
                                     bool store, typename A::V (&v)[kPA]) {
#pragma unroll
    for (int j = 0; j < kPA; j++) {
        v[j] = tile::load_amp(a.in, at(g, gr, j), 0, typename A::V{});
        if (store) A::st(own + slot<A>(j), v[j]);
    }
}

// signs on the register bits zr: at(j) is `one` with bit 31 flipped when j & zr is odd
struct Signs {
    uint32_t lo[4], hi[4];
    __device__ __forceinline__ Signs(uint32_t zr, uint32_t one) {
        const uint32_t s0 = zr << 31, s1 = zr << 30 & 0x80000000u, s2 = zr << 29 & 0x80000000u,
                       s3 = zr << 28 & 0x80000000u;
        lo[0] = one;
        lo[1] = one ^ s0;
        lo[2] = one ^ s1;
        lo[3] = lo[1] ^ s1;
        hi[0] = 0;
        hi[1] = s2;
        hi[2] = s3;
        hi[3] = s2 ^ s3;
    }
    __device__ __forceinline__ float at(int j) const { return __uint_as_float(lo[j & 3] ^ hi[j >> 2 & 3]); }
    __device__ __forceinline__ f2x both(int j) const { return tile::f2x_dup(at(j)); }
};
// x with its sign flipped when z has an odd number of bits
__device__ __forceinline__ uint32_t signed_bits(float x, uint32_t z) {
    return __float_as_uint(x) ^ (uint32_t)__popc(z) << 31;
}

// i v or -i v
__device__ __forceinline__ f2x turned(f2x v, bool plus) { // (-im, re) or (im, -re)
    return f2x_swap(v) ^ (plus ? 0x80000000ull : 0x8000000000000000ull);
}
__device__ __forceinline__ AmpC128::V turned(const AmpC128::V &v, bool plus) {
    return {turned(v.h, plus), turned(v.l, plus)};
}

// a real coefficient on both lanes
struct Coef {
    f2x h, nh, l;
    __device__ __forceinline__ explicit Coef(DF c) : h(tile::f2x_dup(c.hi)), nh(h ^ kSigns), l(tile::f2x_dup(c.lo)) {}
};
__device__ __forceinline__ void mac(f2x &s, const Coef &c, f2x y) { s = f2x_fma(c.h, y, s); }
__device__ __forceinline__ void mac(AmpC128::V &s, const Coef &c, const AmpC128::V &y) {
    tile::pdf_mac(c.h, c.nh, c.l, y.h, y.l, s.h, s.l);
}
// (sh, sl) += c x, x single precision
__device__ __forceinline__ void pdf_mac1(const Coef &c, f2x x, f2x &sh, f2x &sl) {
    const f2x np = tile::f2x_prod(c.nh, x);
    const f2x e = f2x_fma(c.l, x, f2x_fma(c.h, x, np));
    const f2x s = f2x_sub(sh, np);
    const f2x bb = f2x_sub(s, sh);
    const f2x t = f2x_sub(f2x_sub(sh, f2x_sub(s, bb)), f2x_add(np, bb));
    sh = s;
    sl = f2x_add(sl, f2x_add(t, e));
}
// (sh, sl) -= sg a b with sg = +-1 on both lanes; nah = -ah.  The same roundings as
// pdf_mac: sums with a signed product are fused products with +-1.
__device__ __forceinline__ void pdf_msub_signed(f2x ah, f2x nah, f2x al, f2x bh, f2x bl, f2x sg, f2x &sh, f2x &sl) {
    const f2x np = tile::f2x_prod(nah, bh);
    f2x e = f2x_fma(ah, bh, np);
    e = f2x_fma(ah, bl, e);
    e = f2x_fma(al, bh, e);
    const f2x s = f2x_fma(np, sg, sh);
    const f2x nbb = f2x_sub(sh, s);
    const f2x nt = f2x_sub(f2x_sub(f2x_add(s, nbb), sh), f2x_fma(np, sg, nbb));
    sh = s;
    sl = f2x_sub(sl, f2x_fma(e, sg, nt));
}

// High and low part apart again.  An unnormalised low part collects the high
// part's rounding errors and is itself rounded at their size: after n sums the
// error is some n 2^-54 of the sum (a 25-qubit energy of 100 words, one sum per
// thread for all words and tiles: 1.6e-13 of a total of 17).
__device__ __forceinline__ void settle(f2x &h, f2x &l) {
    const f2x s = f2x_add(h, l);
    l = f2x_sub(l, f2x_sub(s, h));
    h = s;
}
__device__ __forceinline__ void settle(f2x &) {}
__device__ __forceinline__ void settle(AmpC128::V &s) { settle(s.h, s.l); }

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

// coefficients of a word group on eight register indices (pairs); top: the upper half
__device__ __forceinline__ void coefficients(const PauliArgs &a, uint32_t many, uint32_t g, uint32_t top, DF (&c)[8]) {
    const uint32_t *off = a.offs + many;
    uint32_t t = off[0];
#pragma unroll
    for (int w = 0; w < 8; w++) {
        c[w] = {0.0f, 0.0f};
        for (const uint32_t end = off[w + 1]; t < end; t++) {
            const Term tt = a.terms[t];
            const bool neg = (__popc(g & tt.z) ^ (tt.top & top)) & 1u;
            df_add(neg ? -tt.ch : tt.ch, neg ? -tt.cl : tt.cl, c[w].hi, c[w].lo);
        }
    }
    walsh<3>(c);
#pragma unroll
    for (int w = 0; w < 8; w++) { // what cancelled may leave a low part as large as the high one
        DF n = {c[w].hi, 0.0f};
        df_add(c[w].lo, 0.0f, n.hi, n.lo);
        c[w] = n;
    }
}

// One word ready to be added: sign and address of a thread's sixteen partners
template <class A> struct Word;
template <> struct Word<AmpC64> {
    uint32_t tx;
    Signs c; // the coefficient, signed by register index
    __device__ __forceinline__ Word(const Item &it, uint32_t g, uint32_t tl)
        : c(it.w >> 16 & 15u, signed_bits(it.ch, g & it.z)) {
        tx = tl * AmpC64::kBytes ^ (it.w & 0xffffu);
    }
    __device__ __forceinline__ void add(f2x &s, int j, const unsigned char *L) const {
        const f2x y = AmpC64::ld(L + (tx ^ slot<AmpC64>(j)));
        const float k = c.at(j); // two scalar products need it once, a packed one twice
        s = f2x_pack(fmaf(k, f2x_lo(y), f2x_lo(s)), fmaf(k, f2x_hi(y), f2x_hi(s)));
    }
};
template <> struct Word<AmpC128> {
    uint32_t tx;
    f2x h, nh, l;
    Signs c;
    __device__ __forceinline__ Word(const Item &it, uint32_t g, uint32_t tl)
        : c(it.w >> 16 & 15u, signed_bits(-1.0f, g & it.z)) {
        tx = tl * AmpC128::kBytes ^ (it.w & 0xffffu);
        h = tile::f2x_dup(it.ch);
        nh = h ^ kSigns;
        l = tile::f2x_dup(it.cl);
    }
    __device__ __forceinline__ void add(AmpC128::V &s, int j, const unsigned char *L) const {
        const AmpC128::V y = AmpC128::ld(L + (tx ^ slot<AmpC128>(j)));
        pdf_msub_signed(h, nh, l, y.h, y.l, c.both(j), s.h, s.l);
    }
};

// items k .. end - 1 added to s: groups of words first, then single words in twos
template <class A>
__device__ __forceinline__ void add_items(const PauliArgs &a, int k, int end, uint32_t g, uint32_t tl,
                                          const unsigned char *L, typename A::V (&s)[kPA]) {
    for (; k < end && a.items[k].w & kMany; k++) {
        const Item it = a.items[k];
        const uint32_t tx = tl * A::kBytes ^ (it.w & 0xffffu);
#pragma unroll
        for (int top = 0; top < 2; top++) {
            DF c[8];
            coefficients(a, it.z, g, top, c);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (A::kBytes == 8) c[i].hi += c[i].lo;
                mac(s[i + 8 * top], Coef(c[i]), A::ld(L + (tx ^ slot<A>(i + 8 * top))));
            }
        }
    }
    if constexpr (A::kBytes == 16) {
        for (; k + 1 < end; k += 2) {
            const Word<A> x(a.items[k], g, tl), y(a.items[k + 1], g, tl);
#pragma unroll
            for (int j = 0; j < kPA; j++) {
                x.add(s[j], j, L);
                y.add(s[j], j, L);
            }
        }
    }
    for (; k < end; k++) {
        const Word<A> x(a.items[k], g, tl);
#pragma unroll
        for (int j = 0; j < kPA; j++) x.add(s[j], j, L);
    }
}

template <int B> constexpr __host__ __device__ int lower(int i) { return B < 4 ? ins0(i, B < 4 ? B : 0) : i; }
template <int B, class V> __device__ __forceinline__ V lower_end(const V (&v)[kPA], int i, bool half) {
    if constexpr (B == 4) return choose(half, v[i | 8], v[i]); // this thread's lower or upper eight
    return v[lower<B>(i)];
}
// c times the lanes of Re conj(a) b summed over eight pairs, signed by zr.
// tx: byte offset of this thread's partners.  complex64 forms the signed sum level
// by level, a product with +-1 each: flipping eight operands keeps the integer
// pipe busier than the sums the FP32 pipe.
template <int B>
__device__ __forceinline__ void pairs(const f2x (&v)[kPA], const unsigned char *L, uint32_t tx, uint32_t zr, bool half,
                                      const Coef &c, f2x &th, f2x &tl) {
    f2x q[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = lower<B>(i);
        q[i] = tile::f2x_prod(lower_end<B>(v, i, half), AmpC64::ld(L + (tx ^ slot<AmpC64>(j))));
    }
#pragma unroll
    for (int b = 0; b < 3; b++) { // pair bit b is register bit b, or b + 1 above bit B
        const f2x sg = tile::f2x_dup(__uint_as_float(0x3f800000u ^ (zr >> (b < B ? b : b + 1) << 31)));
#pragma unroll
        for (int i = 0; i < 4 >> b; i++) q[i] = f2x_fma(q[2 * i + 1], sg, q[2 * i]);
    }
    pdf_mac1(c, q[0], th, tl);
}
template <int B>
__device__ __forceinline__ void pairs(const AmpC128::V (&v)[kPA], const unsigned char *L, uint32_t tx, uint32_t zr,
                                      bool half, const Coef &c, f2x &th, f2x &tl) {
    const Signs sg(zr, __float_as_uint(-1.0f));
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = lower<B>(i);
        const AmpC128::V x = AmpC128::ld(L + (tx ^ slot<AmpC128>(j))), y = lower_end<B>(v, i, half);
        pdf_msub_signed(x.h, x.h ^ kSigns, x.l, y.h, y.l, sg.both(j), sh, sl);
    }
    tile::pdf_mac(c.h, c.nh, c.l, sh, sl, th, tl);
}
__device__ __forceinline__ void weighted(f2x a, f2x b, DF w, f2x &th, f2x &tl) {
    pdf_mac1(Coef(w), tile::f2x_prod(a, b), th, tl);
}
__device__ __forceinline__ void weighted(const AmpC128::V &a, const AmpC128::V &b, DF w, f2x &th, f2x &tl) {
    f2x ph, pl;
    tile::pdf_first(a.h, a.h ^ kSigns, a.l, b.h, b.l, ph, pl);
    const Coef c(w);
    tile::pdf_mac(c.h, c.nh, c.l, ph, pl, th, tl);
}
template <class A, int B>
__device__ __forceinline__ void weighted_pairs(const typename A::V (&v)[kPA], const unsigned char *L, uint32_t tx,
                                               bool half, const DF (&w)[8], f2x &th, f2x &tl) {
#pragma unroll
    for (int i = 0; i < 8; i++)
        weighted(lower_end<B>(v, i, half), A::ld(L + (tx ^ slot<A>(lower<B>(i)))), w[i], th, tl);
}

template <class A> struct Ctas;
template <> struct Ctas<AmpC64> {
    static constexpr int expval = 2, apply = 3;
};
template <> struct Ctas<AmpC128> {
    static constexpr int expval = 2, apply = 2;
};

template <class A>
__device__ __forceinline__ void expval_items(const PauliArgs &a, int k0, int step, uint32_t g, uint32_t tl,
                                             const unsigned char *L, typename A::V (&v)[kPA], f2x &th, f2x &tlo) {
    if (k0 >= a.nitems) return;
    bool turn = true;
    Item it = a.items[k0];
    for (int k = k0; k < a.nitems; k += step) {
        const Item next = a.items[min(k + step, a.nitems - 1)];
        if (turn && k >= a.nreal) {
            turn = false;
#pragma unroll
            for (int j = 0; j < kPA; j++) v[j] = turned(v[j], true);
        }
        uint32_t tx = tl * A::kBytes ^ (it.w & 0xffffu);
        const int p = it.w >> kPairShift & 15u;
        const bool half = p >= kPR && p < kNoPair && (tl >> (p - kPR) & 1u);
        if (half) tx ^= slot<A>(8);
        if (it.w & kMany) {
            DF w[8];
            if (p == kNoPair) {
#pragma unroll
                for (int top = 0; top < 2; top++) {
                    coefficients(a, it.z, g, top, w);
#pragma unroll
                    for (int i = 0; i < 8; i++) weighted(v[i + 8 * top], v[i + 8 * top], w[i], th, tlo);
                }
            } else {
                coefficients(a, it.z, g, half, w);
                switch (p) {
                case 0: weighted_pairs<A, 0>(v, L, tx, half, w, th, tlo); break;
                case 1: weighted_pairs<A, 1>(v, L, tx, half, w, th, tlo); break;
                case 2: weighted_pairs<A, 2>(v, L, tx, half, w, th, tlo); break;
                case 3: weighted_pairs<A, 3>(v, L, tx, half, w, th, tlo); break;
                default: weighted_pairs<A, 4>(v, L, tx, half, w, th, tlo);
                }
            }
        } else {
            const uint32_t zr = it.w >> 16 & 15u;
            const bool neg = (__popc(g & it.z) ^ (half ? zr >> 3 : 0u)) & 1;
            const Coef c(DF{neg ? -it.ch : it.ch, neg ? -it.cl : it.cl});
            switch (p) {
            case 0: pairs<0>(v, L, tx, zr, half, c, th, tlo); break;
            case 1: pairs<1>(v, L, tx, zr, half, c, th, tlo); break;
            case 2: pairs<2>(v, L, tx, zr, half, c, th, tlo); break;
            case 3: pairs<3>(v, L, tx, zr, half, c, th, tlo); break;
            default: pairs<4>(v, L, tx, zr, half, c, th, tlo);
            }
        }
        if (A::kBytes == 16) settle(th, tlo);
        it = next;
    }
}

template <class A>
__global__ void __launch_bounds__(kThreads, Ctas<A>::expval)
    k_pauli_expval_tile(const __grid_constant__ PauliArgs a, double *partials, double *result, unsigned *counter) {
    using V = typename A::V;
    extern __shared__ __align__(16) unsigned char pauli_smem[];
    const int per = 1 << (a.T - kPR);            // threads of the tile
    const int tl = threadIdx.x & (per - 1), grp = threadIdx.x / per, groups = kThreads / per;
    const int cx = blockIdx.x % a.tiles_x, cy = blockIdx.x / a.tiles_x, ny = gridDim.x / a.tiles_x;
    const uint32_t gt = thread_bits(a, tl);
    unsigned char *own = pauli_smem + tl * A::kBytes;
    uint32_t gr[kPR];
#pragma unroll
    for (int i = 0; i < kPR; i++) gr[i] = 1u << a.rpos[i];
    double total = 0.0;
    for (int tile = cx; tile < a.ntiles; tile += a.tiles_x) {
        const uint32_t g = tile_base(a, tile) | gt;
        V v[kPA];
        load<A>(a, g, gr, own, grp == 0, v);
        __syncthreads();
        f2x th = 0, tlo = 0; // lanes (re re, im im)
        expval_items<A>(a, cy * groups + grp, ny * groups, g, tl, pauli_smem, v, th, tlo);
        total += df_join(f2x_lo(th), f2x_lo(tlo)) + df_join(f2x_hi(th), f2x_hi(tlo));
        __syncthreads();
    }
    double acc[1] = {total};
    block_reduce_finish<1>(acc, partials, result, counter);
}

// out (+)= sum over items of c i^ny (-1)^popcount(src & z) in[src], src = m ^ x
template <class A>
__global__ void __launch_bounds__(kThreads, Ctas<A>::apply) k_pauli_apply_tile(const __grid_constant__ PauliArgs a) {
    using V = typename A::V;
    extern __shared__ __align__(16) unsigned char pauli_smem[];
    const int tl = threadIdx.x; // T = kPT
    const uint32_t gt = thread_bits(a, tl);
    uint32_t gr[kPR];
#pragma unroll
    for (int i = 0; i < kPR; i++) gr[i] = 1u << a.rpos[i];
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const uint32_t g = tile_base(a, tile) | gt;
        V s[kPA];
        load<A>(a, g, gr, pauli_smem + tl * A::kBytes, true, s);
#pragma unroll
        for (int j = 0; j < kPA; j++) s[j] = a.accumulate ? tile::load_bits(a.out, at(g, gr, j), V{}) : V{};
        __syncthreads();
#pragma unroll 1
        for (int k = 0, end; k < a.nitems; k = end) { // up to 16 words, without or with a factor i
            end = min(k + 16, k < a.nreal ? a.nreal : a.nitems);
            if (k == a.nreal)
#pragma unroll
                for (int j = 0; j < kPA; j++) s[j] = turned(s[j], false);
            add_items<A>(a, k, end, g, tl, pauli_smem, s);
#pragma unroll
            for (int j = 0; j < kPA; j++) settle(s[j]);
        }
        if (a.nreal < a.nitems)
#pragma unroll
            for (int j = 0; j < kPA; j++) s[j] = turned(s[j], true);
        uint32_t go = g;
        asm volatile("" : "+r"(go)); // the addresses are formed again, not kept in registers
        __syncthreads(); // partners read before the next tile is loaded
#pragma unroll
        for (int j = 0; j < kPA; j++) tile::store_amp(a.out, at(go, gr, j), a.sum_df, s[j]);
    }
}

// --------------------------------------------------------------- host side --
using Pass = PauliTilePass;

struct Plan {
    std::vector<Pass> passes;
    std::vector<Item> items;
    std::vector<Term> terms;
    std::vector<uint32_t> offs;
    std::vector<int> item0; // per pass (and one past)
    std::vector<PauliArgs> args;
};

// The register bits of a pass: those that most X patterns have (a pattern is
// counted once), but not the bits that neighbouring lanes need.
uint32_t choose_register_bits(const Pass &p, int nq, int T, int low, const std::vector<PauliGroup> &groups) {
    const uint32_t keep = T - low >= kPR ? (1u << low) - 1u : 0u;
    uint32_t reg = 0;
    for (int r = 0; r < kPR; r++) {
        int best = -1, most = -1;
        for (int b = nq - 1; b >= 0; b--) {
            if (!(p.bits & ~reg & ~keep & 1u << b)) continue;
            int n = 0;
            for (int gi : p.groups)
                if ((groups[gi].x & reg) == 0 && (groups[gi].x >> b & 1)) n++;
            if (n > most) {
                most = n;
                best = b;
            }
        }
        reg |= 1u << best;
    }
    return reg;
}

// expval: Hermitian form, each pair once
void make_plan(int nq, int dtype, const std::vector<PauliGroup> &groups, const std::vector<PauliTerm> &terms,
               bool expval, Plan &pl, std::vector<PauliGroup> &rest) {
    const bool c64 = dtype == PLK_C64;
    const int T = std::min(kPT, nq), amp = c64 ? 8 : 16;
    const int low = std::min(c64 ? 3 : 2, T);
    const int least = expval ? (c64 ? kManyExpvalC64 : kManyExpvalC128) : (c64 ? kManyApplyC64 : kManyApplyC128);
    choose_passes(nq, T, low, groups, pl.passes, rest);
    if (!expval) keep_worthwhile(ApplyCost(c64, nq), groups, pl.passes, rest);
    for (const Pass &p : pl.passes) {
        PauliArgs a;
        std::memset((void *)&a, 0, sizeof(a));
        a.T = T;
        a.ntiles = 1 << (nq - T);
        const uint32_t reg = choose_register_bits(p, nq, T, low, groups);
        int pos[32], n = 0, nt = 0, nr = 0; // slot bit of a state bit
        for (int b = 0; b < nq; b++) {
            if (!(p.bits >> b & 1)) continue;
            a.gpos[n++] = (uint8_t)b;
            if (reg >> b & 1) {
                pos[b] = kPT - kPR + nr;
                a.rpos[nr++] = (uint8_t)b;
            } else {
                pos[b] = nt;
                a.tpos[nt++] = (uint8_t)b;
            }
        }
        pl.args.push_back(a);
        const size_t first_item = pl.items.size();
        pl.item0.push_back((int)first_item);
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
            const uint32_t xl = local(g.x), xr = xl >> (kPT - kPR);
            const int pair = !xl ? kNoPair : xr ? 31 - __builtin_clz(xr) : kPR + 31 - __builtin_clz(xl);
            for (int odd = 0; odd < 2; odd++) { // c i^ny is real for an even number of Y, imaginary for an odd one
                std::vector<const PauliTerm *> words;
                for (int k = 0; k < g.count; k++)
                    if ((pauli_popc(g.x & terms[g.first + k].z) & 1) == odd) words.push_back(&terms[g.first + k]);
                if (words.empty()) continue;
                const bool many = (int)words.size() >= least || (expval && !g.x);
                // In the expectation value a pair counts twice, and the sign is that of m; applied to m it is that of m ^ x.
                const float scale = expval ? (g.x ? 2.0f : 1.0f) : (odd ? -1.0f : 1.0f);
                const uint32_t w0 = xl * amp | (odd ? kFactorI : 0u) | (uint32_t)pair << kPairShift;
                if (!many) {
                    for (const PauliTerm *t : words) {
                        const uint32_t zr = local(t->z) >> (kPT - kPR);
                        pl.items.push_back({w0 | zr << 16, (uint32_t)t->z, scale * (odd ? t->cih : t->crh),
                                            scale * (odd ? t->cil : t->crl)});
                    }
                    continue;
                }
                pl.items.push_back({w0 | kMany, (uint32_t)pl.offs.size(), 0.0f, 0.0f});
                std::vector<Term> by[8];
                for (const PauliTerm *t : words) {
                    const uint32_t zr = local(t->z) >> (kPT - kPR);
                    // pairs by a register bit: that bit is clear
                    const bool inreg = expval && pair < kPR;
                    const uint32_t w = inreg ? (zr & ((1u << pair) - 1u)) | ((zr >> (pair + 1)) << pair) : zr & 7u;
                    by[w].push_back({(uint32_t)t->z, inreg ? 0u : zr >> 3, scale * (odd ? t->cih : t->crh),
                                     scale * (odd ? t->cil : t->crl)});
                }
                for (const auto &list : by) {
                    pl.offs.push_back((uint32_t)pl.terms.size());
                    pl.terms.insert(pl.terms.end(), list.begin(), list.end());
                }
                pl.offs.push_back((uint32_t)pl.terms.size());
            }
        }
        // without a factor i first, and of each part the groups of words first
        std::stable_sort(pl.items.begin() + first_item, pl.items.end(), [](const Item &x, const Item &y) {
            auto key = [](const Item &t) { return (t.w & kFactorI ? 2 : 0) + (t.w & kMany ? 0 : 1); };
            return key(x) < key(y);
        });
        int nreal = 0;
        for (size_t i = first_item; i < pl.items.size(); i++) nreal += !(pl.items[i].w & kFactorI);
        pl.args.back().nreal = nreal;
    }
    pl.item0.push_back((int)pl.items.size());
}

// items, terms and offsets on the device, in one block of the pool
int upload(const Plan &pl, int device, cudaStream_t st, PoolBuf &buf, PauliArgs &a) {
    DeviceCtx *d = nullptr;
    PLK_TRY(device_ctx(device, &d));
    const size_t bi = sizeof(Item) * pl.items.size(), bt = sizeof(Term) * pl.terms.size(),
                 bo = sizeof(uint32_t) * pl.offs.size();
    std::vector<unsigned char> host(bi + bt + bo + 16);
    if (bi) std::memcpy(host.data(), pl.items.data(), bi);
    if (bt) std::memcpy(host.data() + bi, pl.terms.data(), bt);
    if (bo) std::memcpy(host.data() + bi + bt, pl.offs.data(), bo);
    PLK_CUDA(cudaMallocFromPoolAsync(&buf.p, host.size(), d->pool, st));
    PLK_CUDA(cudaMemcpyAsync(buf.p, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    a.items = buf.as<const Item>();
    a.terms = reinterpret_cast<const Term *>(buf.as<char>() + bi);
    a.offs = reinterpret_cast<const uint32_t *>(buf.as<char>() + bi + bt);
    return PLK_OK;
}

// the slots of a small tile are as far apart as a large one's
size_t smem_of(int dtype) { return (size_t)(dtype == PLK_C64 ? 8 : 16) << kPT; }

// Tiles hold double-float pairs: complex128 with native FP64 arithmetic asked for
// keeps the kernels of expval.cu, whose one-word products are formed in FP64
// (amplitudes of 2^150 and 2^-150 read as 0 here and multiply to 1 there).
bool tiles_allowed(int dtype) { return dtype == PLK_C64 || c128_use_df(); }

template <class K> int opt_in(K kernel, size_t bytes) {
    if (bytes > 48 * 1024) PLK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return PLK_OK;
}

} // namespace

int pauli_tile_expval(plk_state s, const std::vector<PauliGroup> &groups, const std::vector<PauliTerm> &terms,
                      std::vector<PauliGroup> &rest, double &total) {
    total = 0.0;
    if (s->nq < kPR || s->nq > 32 || groups.size() < 2 || !tiles_allowed(s->dtype)) {
        rest = groups;
        return PLK_OK;
    }
    Plan pl;
    make_plan(s->nq, s->dtype, groups, terms, true, pl, rest);
    if (pl.passes.empty()) return PLK_OK;
    PoolBuf buf(s->stream);
    PauliArgs dev;
    PLK_TRY(upload(pl, s->device, s->stream, buf, dev));
    const bool c64 = s->dtype == PLK_C64;
    const int T = pl.args[0].T;
    const size_t smem = smem_of(s->dtype);
    PLK_TRY(c64 ? opt_in(k_pauli_expval_tile<AmpC64>, smem) : opt_in(k_pauli_expval_tile<AmpC128>, smem));
    const int cap = device_sm_count(s->device) * (c64 ? Ctas<AmpC64>::expval : Ctas<AmpC128>::expval);
    const int groups_in_cta = kThreads >> (T - kPR);
    auto &w = s->ws;
    std::vector<double> vals(pl.passes.size());
    for (size_t i = 0; i < pl.passes.size(); i++) {
        PauliArgs a = pl.args[i];
        a.in = s->data;
        a.items = dev.items + pl.item0[i];
        a.terms = dev.terms;
        a.offs = dev.offs;
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
    accumulate = false;
    // below 18 qubits the plain kernel was ahead wherever it was measured (40 words of
    // weight 8, us on tiles / plain: 13 qubits complex64 49 / 40, 16 qubits 44 / 40)
    if (out->nq < 18 || out->nq > 32 || groups.size() < 2 || !tiles_allowed(out->dtype) ||
        !ApplyCost(out->dtype == PLK_C64, out->nq).worth_a_look(groups)) {
        rest = groups;
        return PLK_OK;
    }
    Plan pl;
    make_plan(out->nq, out->dtype, groups, terms, false, pl, rest);
    if (pl.passes.empty()) return PLK_OK;
    cudaStream_t st = out->stream;
    PoolBuf buf(st);
    PauliArgs dev;
    PLK_TRY(upload(pl, out->device, st, buf, dev));
    const bool c64 = out->dtype == PLK_C64;
    const size_t smem = smem_of(out->dtype);
    PLK_TRY(c64 ? opt_in(k_pauli_apply_tile<AmpC64>, smem) : opt_in(k_pauli_apply_tile<AmpC128>, smem));
    const int cap = device_sm_count(out->device) * (c64 ? Ctas<AmpC64>::apply : Ctas<AmpC128>::apply);
    for (size_t i = 0; i < pl.passes.size(); i++) {
        PauliArgs a = pl.args[i];
        a.in = in->data;
        a.out = out->data;
        a.items = dev.items + pl.item0[i];
        a.terms = dev.terms;
        a.offs = dev.offs;
        a.nitems = pl.item0[i + 1] - pl.item0[i];
        a.accumulate = accumulate;
        a.sum_df = i + 1 < pl.passes.size();
        const int grid = std::min(a.ntiles, cap);
        if (c64) k_pauli_apply_tile<AmpC64><<<grid, kThreads, smem, st>>>(a);
        else k_pauli_apply_tile<AmpC128><<<grid, kThreads, smem, st>>>(a);
        PLK_CHECK_LAUNCH();
        accumulate = true;
    }
    return PLK_OK;
}

} // namespace plk
