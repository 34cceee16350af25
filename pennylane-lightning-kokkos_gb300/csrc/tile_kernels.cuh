// tile_kernels.cuh — device side of the tile sweeps (programs: tile_program.hpp).
//
// A CTA works on a tile of 2^T amplitudes (of lambda, and of H lambda going
// backwards) at a time, in rounds: a thread holds the 2^R amplitudes that differ
// in the round's R register bits in registers and runs the round's stages on
// them with compile-time register indices.  The first round reads the state, the
// last one writes it; in between the amplitudes go through shared memory, each
// thread writing to the slots it has just read, with one barrier per round.
// CNOTs, X and SWAP cost nothing: the rounds' slot maps carry them.  Slots are
// XOR-swizzled and the host picks lane bits whose slots fall into different
// banks.
//
// complex64 runs a rotation as three shears, x -= t y, y += s x, x -= t y with
// t = tan(angle / 2) <= 0.42: every step updates a register in place, so the
// branches around a step need no register moves (the two-output form cost one
// move per amplitude and step, a quarter of all instructions).  complex128 is
// bound by the FP32 pipe, where a product and sum of double-floats takes 12
// packed instructions: it runs [[1, -t], [t, 1]], two of them per pair, and
// leaves the cosine to the next phase table.
//
// complex64: an amplitude is one packed FP32 pair (re, im), so a rotation is
// three .f32x2 instructions per pair of amplitudes.  complex128: the tile holds
// double-float amplitudes as two packed pairs, (re.hi, im.hi) and
// (re.lo, im.lo), for the whole sweep; arithmetic as in df.cuh.
//
// Sums for gradients (Im <h|X|v>, Im <h|Y|v>, Walsh sums of Im(conj h v)) are
// formed per thread (complex64: eight products in FP32, then double-float;
// complex128: double-float), reduced over the warp in a fixed pattern after
// each stage and kept per warp in shared memory as double-floats: reruns are
// bitwise identical.  A tile of fewer amplitudes than a warp holds is worked on
// by several lanes alike; the host scales its sums.
#pragma once

#include "df.cuh"
#include "plk_internal.cuh"
#include "tile_program.hpp"

namespace plk {
namespace tile {

// gridDim.y sweeps share the program: sweep y reads lam_src[y] and writes
// lam[y] (the same buffer after the first pass), and works on hl[y] in place.
constexpr int kMaxSweeps = 32;
struct Args {
    const void *lam_src[kMaxSweeps];
    void *lam[kMaxSweeps], *hl[kMaxSweeps];
    const unsigned char *prog; // this pass's blob
    uint32_t prog_bytes;
    int T, nacc, ntiles;
    int nacc_all;      // accumulators of the whole program
    int in_df, out_df; // complex128: buffers hold doubles (0) or double-float pairs (1) on entry / exit, or
                       // doubles that a program of index maps alone moves as they are (2)
    int drop;          // the states on exit are not wanted
    double *part;      // [sweep][accumulator][gridDim.x]
    // when set, H lambda of sweep y starts as the Pauli word i^ny (-1)^popcount(k & z) |k ^ x> on lam_src[y]
    int words;
    uint32_t wx[kMaxSweeps], wz[kMaxSweeps];
    uint8_t wq[kMaxSweeps]; // number of Y letters
};

__device__ __forceinline__ f2x f2x_dup(float a) { return f2x_pack(a, a); }
__device__ __forceinline__ float f2x_lo(f2x v) {
    float a, b;
    f2x_unpack(v, a, b);
    return a;
}
__device__ __forceinline__ float f2x_hi(f2x v) {
    float a, b;
    f2x_unpack(v, a, b);
    return b;
}

// ---- packed double-float with one negated operand -------------------------
// np = -(a * b) lets the error term and the difference p - bb be formed without
// negating data: only nah = -ah is needed.  Products are rounded by an fma with
// zero: mul.rn.f32x2 feeding sub.rn.f32x2 was contracted (a product followed by
// the sum below lost half the bits), an fma cannot be.
__device__ __forceinline__ f2x f2x_prod(f2x a, f2x b) { return f2x_fma(a, b, 0ull); }
__device__ __forceinline__ void pdf_mac(f2x ah, f2x nah, f2x al, f2x bh, f2x bl, f2x &sh, f2x &sl) {
    const f2x np = f2x_prod(nah, bh);
    f2x e = f2x_fma(ah, bh, np);
    e = f2x_fma(ah, bl, e);
    e = f2x_fma(al, bh, e);
    const f2x s = f2x_sub(sh, np);
    const f2x bb = f2x_sub(s, sh);
    const f2x t = f2x_sub(f2x_sub(sh, f2x_sub(s, bb)), f2x_add(np, bb));
    sh = s;
    sl = f2x_add(sl, f2x_add(t, e));
}
// (sh, sl) -= a * b
__device__ __forceinline__ void pdf_msub(f2x ah, f2x nah, f2x al, f2x bh, f2x bl, f2x &sh, f2x &sl) {
    const f2x np = f2x_prod(nah, bh);
    f2x e = f2x_fma(ah, bh, np);
    e = f2x_fma(ah, bl, e);
    e = f2x_fma(al, bh, e);
    const f2x s = f2x_add(sh, np);
    const f2x bb = f2x_sub(s, sh);
    const f2x t = f2x_add(f2x_sub(sh, f2x_sub(s, bb)), f2x_sub(np, bb));
    sh = s;
    sl = f2x_add(sl, f2x_sub(t, e));
}
__device__ __forceinline__ void pdf_first(f2x ah, f2x nah, f2x al, f2x bh, f2x bl, f2x &sh, f2x &sl) {
    sh = f2x_prod(ah, bh);
    f2x e = f2x_fma(ah, bh, f2x_prod(nah, bh));
    e = f2x_fma(ah, bl, e);
    sl = f2x_fma(al, bh, e);
}

// ------------------------------------------------------------ amplitudes ----
struct AmpC64 {
    static constexpr int kBytes = 8;
    using V = f2x;
    static __device__ __forceinline__ V ld(const unsigned char *p) { return *reinterpret_cast<const f2x *>(p); }
    static __device__ __forceinline__ void st(unsigned char *p, const V &v) { *reinterpret_cast<f2x *>(p) = v; }
};
struct AmpC128 {
    static constexpr int kBytes = 16;
    struct V {
        f2x h, l;
    };
    static __device__ __forceinline__ V ld(const unsigned char *p) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p);
        return {a.x, a.y};
    }
    static __device__ __forceinline__ void st(unsigned char *p, const V &v) {
        *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.h, v.l);
    }
};

// x -= t y, y += s x, x -= t y
struct RotC64 {
    f2x nt, s;
    __device__ __forceinline__ explicit RotC64(float4 k) : nt(f2x_dup(-k.x)), s(f2x_dup(k.z)) {}
    __device__ __forceinline__ void operator()(f2x &x, f2x &y) const {
        x = f2x_fma(nt, y, x);
        y = f2x_fma(s, x, y);
        x = f2x_fma(nt, y, x);
    }
};
// (x, y) <- (x - t y, y + t x); the factor cos is in a phase table
struct RotC128 {
    f2x th, nth, tl;
    __device__ __forceinline__ explicit RotC128(float4 k) : th(f2x_dup(k.x)), nth(f2x_dup(-k.x)), tl(f2x_dup(k.y)) {}
    __device__ __forceinline__ void operator()(AmpC128::V &x, AmpC128::V &y) const {
        const AmpC128::V x0 = x;
        pdf_msub(th, nth, tl, y.h, y.l, x.h, x.l);
        pdf_mac(th, nth, tl, x0.h, x0.l, y.h, y.l);
    }
};
// (x, y) <- (c x - s y, s x + c y): any angle, and exact for quarter turns
struct TurnC64 {
    f2x c, s, ns;
    __device__ __forceinline__ explicit TurnC64(float4 k) : c(f2x_dup(k.x)), s(f2x_dup(k.z)), ns(f2x_dup(-k.z)) {}
    __device__ __forceinline__ void operator()(f2x &x, f2x &y) const {
        const f2x nx = f2x_fma(ns, y, f2x_mul(c, x));
        y = f2x_fma(s, x, f2x_mul(c, y));
        x = nx;
    }
};
struct TurnC128 {
    f2x ch, nch, cl, sh, nsh, sl;
    __device__ __forceinline__ explicit TurnC128(float4 k)
        : ch(f2x_dup(k.x)), nch(f2x_dup(-k.x)), cl(f2x_dup(k.y)), sh(f2x_dup(k.z)), nsh(f2x_dup(-k.z)),
          sl(f2x_dup(k.w)) {}
    __device__ __forceinline__ void operator()(AmpC128::V &x, AmpC128::V &y) const {
        AmpC128::V a, b;
        pdf_first(ch, nch, cl, x.h, x.l, a.h, a.l);
        pdf_msub(sh, nsh, sl, y.h, y.l, a.h, a.l);
        pdf_first(ch, nch, cl, y.h, y.l, b.h, b.l);
        pdf_mac(sh, nsh, sl, x.h, x.l, b.h, b.l);
        x = a;
        y = b;
    }
};

template <class A> struct Form;
template <> struct Form<AmpC64> {
    using Rot = RotC64;
    using Turn = TurnC64;
    using E = float2; // table entry: re im
};
template <> struct Form<AmpC128> {
    using Rot = RotC128;
    using Turn = TurnC128;
    using E = float4; // re.hi im.hi re.lo im.lo
};

constexpr __host__ __device__ int ins0(int p, int b) { return ((p >> b) << (b + 1)) | (p & ((1 << b) - 1)); }

// double-float (h, l) += x, both lanes
__device__ __forceinline__ void f2x_addf(f2x x, f2x &h, f2x &l) {
    const f2x s = f2x_add(h, x);
    const f2x bb = f2x_sub(s, h);
    const f2x t = f2x_add(f2x_sub(h, f2x_sub(s, bb)), f2x_sub(x, bb));
    h = s;
    l = f2x_add(l, t);
}
__device__ __forceinline__ DF f2x_total(f2x h, f2x l) { // lane 0 + lane 1
    DF r = {f2x_lo(h), f2x_lo(l)};
    df_add(f2x_hi(h), f2x_hi(l), r.hi, r.lo);
    return r;
}

// Im <h|Y|v> = Re(conj(h1) v0) - Re(conj(h0) v1) over the active pairs of bit
// B.  complex64: four pairs in FP32 per lane (eight products), then
// double-float.
template <int NA, int B, bool CTRL>
__device__ __forceinline__ DF sum_y(const f2x (&v)[NA], const f2x (&h)[NA], uint32_t act) {
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int q = 0; q < NA / 2; q += 4) {
        f2x p = 0, m = 0;
#pragma unroll
        for (int i = q; i < q + 4; i++) {
            const int a = ins0(i, B), b = a | 1 << B;
            if (CTRL && !(act >> a & 1)) continue;
            p = f2x_fma(h[b], v[a], p);
            m = f2x_fma(h[a], v[b], m);
        }
        f2x_addf(f2x_sub(p, m), sh, sl);
    }
    return f2x_total(sh, sl);
}
template <int NA, int B, bool CTRL>
__device__ __forceinline__ DF sum_y(const AmpC128::V (&v)[NA], const AmpC128::V (&h)[NA], uint32_t act) {
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int i = 0; i < NA / 2; i++) {
        const int a = ins0(i, B), b = a | 1 << B;
        if (CTRL && !(act >> a & 1)) continue;
        pdf_mac(h[b].h, f2x_sub(0ull, h[b].h), h[b].l, v[a].h, v[a].l, sh, sl);
        pdf_msub(h[a].h, f2x_sub(0ull, h[a].h), h[a].l, v[b].h, v[b].l, sh, sl);
    }
    return f2x_total(sh, sl);
}
// Im <h|X|v> = Im(conj(h0) v1) + Im(conj(h1) v0); lanes (h.re v.im, h.im v.re),
// whose difference is Im(conj h v)
template <int NA, int B> __device__ __forceinline__ DF sum_x(const f2x (&v)[NA], const f2x (&h)[NA]) {
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int q = 0; q < NA / 2; q += 4) {
        f2x p = 0;
#pragma unroll
        for (int i = q; i < q + 4; i++) {
            const int a = ins0(i, B), b = a | 1 << B;
            p = f2x_fma(h[a], f2x_swap(v[b]), p);
            p = f2x_fma(h[b], f2x_swap(v[a]), p);
        }
        f2x_addf(p, sh, sl);
    }
    DF r = {f2x_lo(sh), f2x_lo(sl)};
    df_add(-f2x_hi(sh), -f2x_hi(sl), r.hi, r.lo);
    return r;
}
template <int NA, int B> __device__ __forceinline__ DF sum_x(const AmpC128::V (&v)[NA], const AmpC128::V (&h)[NA]) {
    f2x sh = 0, sl = 0;
#pragma unroll
    for (int i = 0; i < NA / 2; i++) {
        const int a = ins0(i, B), b = a | 1 << B;
        pdf_mac(h[a].h, f2x_sub(0ull, h[a].h), h[a].l, f2x_swap(v[b].h), f2x_swap(v[b].l), sh, sl);
        pdf_mac(h[b].h, f2x_sub(0ull, h[b].h), h[b].l, f2x_swap(v[a].h), f2x_swap(v[a].l), sh, sl);
    }
    DF r = {f2x_lo(sh), f2x_lo(sl)};
    df_add(-f2x_hi(sh), -f2x_hi(sl), r.hi, r.lo);
    return r;
}

// v <- e v
__device__ __forceinline__ void phase(f2x &v, float2 e) {
    float a, b;
    f2x_unpack(v, a, b);
    v = f2x_pack(fmaf(a, e.x, -b * e.y), fmaf(a, e.y, b * e.x));
}
__device__ __forceinline__ void phase(AmpC128::V &v, float4 e) {
    float ah, bh, al, bl;
    f2x_unpack(v.h, ah, bh);
    f2x_unpack(v.l, al, bl);
    float rh, rl, ih, il;
    df_first(e.x, e.z, ah, al, rh, rl);
    df_mac(-e.y, -e.w, bh, bl, rh, rl);
    df_first(e.x, e.z, bh, bl, ih, il);
    df_mac(e.y, e.w, ah, al, ih, il);
    v.h = f2x_pack(rh, ih);
    v.l = f2x_pack(rl, il);
}

// Im(conj(h) v): complex64 in FP32 (low part 0), complex128 in double-float
__device__ __forceinline__ DF im_dot(f2x h, f2x v) {
    float a, b, c, d;
    f2x_unpack(h, a, b);
    f2x_unpack(v, c, d);
    return {fmaf(a, d, -b * c), 0.0f};
}
__device__ __forceinline__ DF im_dot(const AmpC128::V &h, const AmpC128::V &v) {
    float ah, bh, al, bl, ch, dh, cl, dl, rh, rl;
    f2x_unpack(h.h, ah, bh);
    f2x_unpack(h.l, al, bl);
    f2x_unpack(v.h, ch, dh);
    f2x_unpack(v.l, cl, dl);
    df_first(ah, al, dh, dl, rh, rl);
    df_mac(-bh, -bl, ch, cl, rh, rl);
    return {rh, rl};
}
template <class A> __device__ __forceinline__ DF c_add(DF a, DF b) {
    if constexpr (A::kBytes == 8) return {a.hi + b.hi, 0.0f};
    df_add(b.hi, b.lo, a.hi, a.lo);
    return a;
}
template <class A> __device__ __forceinline__ DF c_sub(DF a, DF b) {
    if constexpr (A::kBytes == 8) return {a.hi - b.hi, 0.0f};
    df_add(-b.hi, -b.lo, a.hi, a.lo);
    return a;
}

// sum of a value over the warp (every lane)
__device__ __forceinline__ DF warp_sum(DF a) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, a.hi, o), ol = __shfl_xor_sync(0xffffffffu, a.lo, o);
        df_add(oh, ol, a.hi, a.lo);
    }
    return a;
}
__device__ __forceinline__ void acc_add(float2 *row, int id, DF v) {
    float2 a = row[id];
    df_add(v.hi, v.lo, a.x, a.y);
    row[id] = a;
}
__device__ __forceinline__ DF shfl(DF a, int o) {
    return {__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}
__device__ __forceinline__ DF pick(bool c, DF a, DF b) { return {c ? a.hi : b.hi, c ? a.lo : b.lo}; }
__device__ __forceinline__ DF plus(DF a, DF b) {
    df_add(b.hi, b.lo, a.hi, a.lo);
    return a;
}
__device__ __forceinline__ f2x shfl(f2x a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
// Sums of N = 4 or 8 values over the warp.  Each of the first exchanges halves the
// number of values a lane carries (eight sums take 9 exchanges instead of 40), two
// values to an instruction while there are two.  The lane ends up with value k.
template <int N> __device__ __forceinline__ DF warp_sums(const DF (&x)[N], int lane, int &k) {
    f2x h[N / 2], l[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        h[i] = f2x_pack(x[2 * i].hi, x[2 * i + 1].hi);
        l[i] = f2x_pack(x[2 * i].lo, x[2 * i + 1].lo);
    }
    k = 0;
    int o = 16;
#pragma unroll
    for (int n = N / 4; n; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const f2x ah = up ? h[i] : h[i + n], al = up ? l[i] : l[i + n];
            if (up) {
                h[i] = h[i + n];
                l[i] = l[i + n];
            }
            const f2x bh = shfl(ah, o), s = f2x_add(h[i], bh), bb = f2x_sub(s, h[i]);
            const f2x t = f2x_add(f2x_sub(h[i], f2x_sub(s, bb)), f2x_sub(bh, bb));
            l[i] = f2x_add(l[i], f2x_add(t, shfl(al, o)));
            h[i] = s;
        }
        k += up ? 2 * n : 0;
    }
    const bool up = lane & o;
    const DF a = {f2x_lo(h[0]), f2x_lo(l[0])}, b = {f2x_hi(h[0]), f2x_hi(l[0])};
    DF t = plus(pick(up, b, a), shfl(pick(up, a, b), o));
    k += up ? 1 : 0;
#pragma unroll
    for (int q = 16 / N; q; q >>= 1) t = plus(t, shfl(t, q));
    return t;
}
// the warp's sums added to accumulators, `mine` for the value this lane has (-1: none)
template <int N> __device__ __forceinline__ void acc_sums(float2 *row, int lane, int mine, DF t) {
    if ((lane & (32 / N - 1)) == 0 && mine >= 0) acc_add(row, mine, t);
}

// Walsh sums of c_j = Im(conj h_j v_j) over single register bits, through a tree
template <class A, int R>
__device__ __forceinline__ void walsh_bits(const typename A::V (&v)[1 << R], const typename A::V (&h)[1 << R], DF *z) {
    constexpr int NA = 1 << R;
    DF c[NA / 2], d = {0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < NA / 2; k++) {
        const DF a = im_dot(h[2 * k], v[2 * k]), b = im_dot(h[2 * k + 1], v[2 * k + 1]);
        const DF e = c_sub<A>(a, b);
        d = k ? c_add<A>(d, e) : e;
        c[k] = c_add<A>(a, b);
    }
    z[0] = d;
#pragma unroll
    for (int b = 1; b < R; b++) {
#pragma unroll
        for (int k = 0; k < (NA / 2) >> b; k++) {
            const DF e = c_sub<A>(c[2 * k], c[2 * k + 1]);
            d = k ? c_add<A>(d, e) : e;
            c[k] = c_add<A>(c[2 * k], c[2 * k + 1]);
        }
        z[b] = d;
    }
}

// any masks, through the full transform
template <class A, int R>
__device__ __forceinline__ void walsh_all(const typename A::V (&v)[1 << R], const typename A::V (&h)[1 << R],
                                          uint32_t zsel, int next, float2 *row, int lane) {
    constexpr int NA = 1 << R;
    DF c[NA];
#pragma unroll
    for (int j = 0; j < NA; j++) c[j] = im_dot(h[j], v[j]);
#pragma unroll
    for (int b = 0; b < R; b++)
#pragma unroll
        for (int p = 0; p < NA / 2; p++) {
            const int i = ins0(p, b), k = i | 1 << b;
            const DF s = c_add<A>(c[i], c[k]);
            c[k] = c_sub<A>(c[i], c[k]);
            c[i] = s;
        }
#pragma unroll
    for (int g = 0; g < NA / 4; g++)
        if (zsel >> (4 * g) & 15u) {
            DF x[4];
#pragma unroll
            for (int m = 0; m < 4; m++) x[m] = c[4 * g + m];
            const uint32_t z = zsel >> (4 * g) & 15u;
            int k;
            const DF t = warp_sums<4>(x, lane, k);
            acc_sums<4>(row, lane, z >> k & 1 ? next + __popc(z & ((1u << k) - 1u)) : -1, t);
            next += __popc(z);
        }
}

// A diagonal step whose phase needs the state index of each amplitude.
template <class A, int R, bool BWD>
__device__ __forceinline__ void step_index(typename A::V (&v)[1 << R], typename A::V (&h)[1 << R], const TileStage &st,
                                           const TileIndex &x, uint32_t gi, const unsigned char *tab, float2 *row,
                                           int lane) {
    const auto *e = reinterpret_cast<const typename Form<A>::E *>(tab) + st.stab;
    const bool par = st.special == TS_PAR, gr = BWD && st.sacc >= 0;
    uint32_t f0 = 0, fr[4] = {0, 0, 0, 0}; // table index of the thread's part, flips of each register bit
    if (par) {
        f0 = __popc(gi & st.cmask) & 1;
#pragma unroll
        for (int i = 0; i < R; i++) fr[i] = (x.r[i] & st.cmask) ? 1u : 0u;
    } else {
        for (int q = 0; q < st.K; q++) {
            const uint32_t b = st.cmask >> (5 * q) & 31u;
            f0 |= (gi >> b & 1u) << q;
#pragma unroll
            for (int i = 0; i < R; i++)
                if (x.r[i] == 1u << b) fr[i] = 1u << q;
        }
    }
    DF a = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 1 << R; j++) {
        const uint32_t f = f0 ^ ((j & 1) ? fr[0] : 0) ^ ((j & 2) ? fr[1] : 0) ^ ((j & 4) ? fr[2] : 0) ^
                           ((j & 8) ? fr[3] : 0);
        if (gr) {
            const float g = par ? (f ? -1.0f : 1.0f) : reinterpret_cast<const float *>(tab)[st.gtab + f];
            const DF c = im_dot(h[j], v[j]);
            df_add(g * c.hi, g * c.lo, a.hi, a.lo); // g is 0 or +-1
        }
        const auto z = e[f];
        phase(v[j], z);
        if (BWD) phase(h[j], z);
    }
    if (gr) {
        a = warp_sum(a);
        if (lane == 0) acc_add(row, st.sacc, a);
    }
}

// Rotation of register bit B: sums first (both states as they are before it)
template <class A, int R, bool BWD, int B>
__device__ __forceinline__ void step_ry(typename A::V (&v)[1 << R], typename A::V (&h)[1 << R], const TileStage &st,
                                        uint32_t ry, DF (&y)[4], DF (&x)[4]) {
    if constexpr (B < R) {
        if (!(ry >> B & 1)) return;
        if (BWD) {
            if (st.acc_y[B] >= 0) y[B] = sum_y<1 << R, B, false>(v, h, 0u);
            if (st.acc_x[B] >= 0) x[B] = sum_x<1 << R, B>(v, h);
        }
        const typename Form<A>::Rot rot(*reinterpret_cast<const float4 *>(st.rot[B]));
#pragma unroll
        for (int p = 0; p < 1 << (R - 1); p++) {
            const int a = ins0(p, B), b = a | 1 << B;
            rot(v[a], v[b]);
            if (BWD) rot(h[a], h[b]);
        }
    }
}

template <class A, int R, bool BWD, int B>
__device__ __forceinline__ void step_cry(typename A::V (&v)[1 << R], typename A::V (&h)[1 << R], const TileStage &st,
                                         uint32_t act, DF &y) {
    if constexpr (B < R) {
        if (BWD && st.sacc >= 0) y = sum_y<1 << R, B, true>(v, h, act);
        const typename Form<A>::Turn turn(*reinterpret_cast<const float4 *>(st.coef));
#pragma unroll
        for (int p = 0; p < 1 << (R - 1); p++) {
            const int a = ins0(p, B), b = a | 1 << B;
            if (!(act >> a & 1)) continue;
            turn(v[a], v[b]);
            if (BWD) turn(h[a], h[b]);
        }
    }
}

// A double as a normalised double-float, both parts rounded to nearest.  The
// truncating split of df.cuh leaves a low part of up to 2^-23 of the high part,
// always of its sign, and what it cuts off and the low parts' dropped products
// add up to a bias of about 2^-48 of a sum's magnitudes (seen in energies whose
// words nearly cancel: 8e-13 against 8e-14).  A float's exponent is the double's
// less 896, which is its low eight bits with the top one flipped; the 29 bits that
// the high part leaves out are converted as an integer and scaled by the high
// part's power of two.  (Assembled from shifted fields on the integer pipe the
// split took twice the instructions, a third of a pass over a Pauli sum.)
__device__ __forceinline__ DF df_split_near(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const unsigned hw = (unsigned)(u >> 32), lw = (unsigned)u;
    const unsigned mag = (__funnelshift_l(lw, hw, 3) ^ 0x40000000u) & 0x7fffffffu;
    const bool fits = 2u * hw - (897u << 21) < (254u << 21); // a normal float; else 0
    const float hi = fits ? __uint_as_float(mag | (hw & 0x80000000u)) : 0.0f;
    const float power = __uint_as_float(__float_as_uint(hi) & 0xff800000u);
    const float lo = __fmul_rn(__fmul_rn(__uint2float_rn(lw & 0x1fffffffu), 0x1p-52f), power);
    const float s = __fadd_rn(hi, lo);
    return {s, __fsub_rn(lo, __fsub_rn(s, hi))};
}

// state buffers: complex128 holds doubles outside a sweep and double-float
// pairs between its passes
__device__ __forceinline__ f2x load_bits(const void *p, uint32_t i, f2x) {
    return __ldcg(static_cast<const unsigned long long *>(p) + i);
}
__device__ __forceinline__ AmpC128::V load_bits(const void *p, uint32_t i, AmpC128::V) {
    const ulonglong2 a = __ldcg(static_cast<const ulonglong2 *>(p) + i);
    return {a.x, a.y};
}
__device__ __forceinline__ f2x from_bits(f2x v) { return v; }
__device__ __forceinline__ AmpC128::V from_bits(const AmpC128::V &v) { // of doubles
    const DF re = df_split_near(__longlong_as_double((long long)v.h));
    const DF im = df_split_near(__longlong_as_double((long long)v.l));
    return {f2x_pack(re.hi, im.hi), f2x_pack(re.lo, im.lo)};
}
template <class V> __device__ __forceinline__ V load_amp(const void *p, uint32_t i, int df, V) {
    const V v = load_bits(p, i, V{});
    return df ? v : from_bits(v);
}
// amplitude i of |0...0>
__device__ __forceinline__ f2x basis_amp(uint32_t i, f2x) { return f2x_pack(i == 0 ? 1.0f : 0.0f, 0.0f); }
__device__ __forceinline__ AmpC128::V basis_amp(uint32_t i, AmpC128::V) {
    return {f2x_pack(i == 0 ? 1.0f : 0.0f, 0.0f), 0ull};
}
__device__ __forceinline__ void store_amp(void *p, uint32_t i, int, f2x v) {
    __stcg(static_cast<unsigned long long *>(p) + i, v);
}
// Between passes the high and low parts are set apart again: rotations leave the
// low part unnormalised, it collects rounding errors and is itself rounded at
// their size (state errors over a list of gates: 1.9e-13 without, 6e-14 with).
__device__ __forceinline__ void store_amp(void *p, uint32_t i, int df, AmpC128::V v) {
    if (df == 1) {
        const f2x s = f2x_add(v.h, v.l);
        v.l = f2x_sub(v.l, f2x_sub(s, v.h));
        v.h = s;
    } else if (df == 0) {
        const double re = df_join(f2x_lo(v.h), f2x_lo(v.l)), im = df_join(f2x_hi(v.h), f2x_hi(v.l));
        v = {(f2x)__double_as_longlong(re), (f2x)__double_as_longlong(im)};
    }
    __stcg(static_cast<ulonglong2 *>(p) + i, make_ulonglong2(v.h, v.l));
}

// A pass's blob in shared memory
struct Pass {
    const TileHdr &hd;
    const TileRound *rounds;
    const TileStage *stages;
    const TileEvent *events;
    const TileIndex *index;
    const unsigned char *tab;
    __device__ __forceinline__ explicit Pass(const unsigned char *p)
        : hd(*reinterpret_cast<const TileHdr *>(p)),
          rounds(reinterpret_cast<const TileRound *>(p + hd.off_rounds)),
          stages(reinterpret_cast<const TileStage *>(p + hd.off_stages)),
          events(reinterpret_cast<const TileEvent *>(p + hd.off_events)),
          index(reinterpret_cast<const TileIndex *>(p + hd.off_index)), tab(p + hd.off_tab) {}
};

// The fields of a stage and a round that every thread needs, in one shared-memory
// read each: read one by one, each branch waited for its own.
struct StageHead {
    uint32_t ry, table, special, sums, tab, zsel;
    int acc_z;
    __device__ __forceinline__ explicit StageHead(const TileStage &st) {
        const uint4 w = *reinterpret_cast<const uint4 *>(&st.ry);
        ry = w.x & 255u;
        table = w.x >> 8 & 255u;
        special = w.x >> 16 & 255u;
        sums = w.x >> 24;
        tab = w.y & 0xffffu;
        zsel = w.y >> 16;
        acc_z = (int16_t)(w.z & 0xffffu);
    }
};
struct RoundHead {
    uint32_t r0, r1, r2, r3, xorc, stage0, nstages, ev0;
    __device__ __forceinline__ explicit RoundHead(const TileRound &q) {
        const uint4 w = *reinterpret_cast<const uint4 *>(q.rcol);
        r0 = w.x & 0xffffu;
        r1 = w.x >> 16;
        r2 = w.y & 0xffffu;
        r3 = w.y >> 16;
        xorc = w.z & 0xffffu;
        stage0 = w.z >> 16;
        nstages = w.w & 0xffffu;
        ev0 = w.w >> 16;
    }
};

// state buffers of a sweep
struct Buffers {
    const void *lam_src;
    void *lam, *hl;
    int in_df, out_df; // complex128: what the buffers hold on entry / exit, as in Args
    bool from_zero;    // the state is |0...0> on entry, lam_src is not read
    bool drop;         // the states on exit are not written: a backward sweep's last pass on buffers of its own
                       // (Jacobian of 20 observables on 20 qubits complex128 30.21 -> 30.06 ms)
    bool word;         // H lambda is a Pauli word on lam_src, hl is not read
    uint32_t wx, wz, wq;
};

// All rounds of one tile; every thread of the CTA takes part.  L, M: the tile's
// slots of lambda and H lambda; row: this warp's accumulators.
__device__ __forceinline__ f2x times_i(f2x v) { return f2x_pack(-f2x_hi(v), f2x_lo(v)); }
__device__ __forceinline__ AmpC128::V times_i(const AmpC128::V &v) { return {times_i(v.h), times_i(v.l)}; }
__device__ __forceinline__ f2x negate(f2x v) { return v ^ 0x8000000080000000ull; }
__device__ __forceinline__ AmpC128::V negate(const AmpC128::V &v) { return {negate(v.h), negate(v.l)}; }

template <class A, int R, bool BWD>
__device__ __forceinline__ void run_tile(const Pass &ps, const Buffers &bf, int tile, int T, unsigned char *L,
                                         unsigned char *M, float2 *row) {
    using V = typename A::V;
    constexpr int NA = 1 << R;
    const TileHdr &hd = ps.hd;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nrounds = hd.nrounds;
    uint32_t base = (uint32_t)tile;
    for (int k = 0; k < T; k++) {
        const uint32_t lo = base & ((1u << hd.gpos[k]) - 1u);
        base = ((base ^ lo) << 1) | lo;
    }
    uint32_t ev = 0;
    for (int r = 0; r < nrounds; r++) {
        const TileRound &q = ps.rounds[r];
        const RoundHead rh(q);
        uint32_t gev = base;
        for (int k = 0; k < q.nev; k++)
            if (base >> ps.events[rh.ev0 + k].bit & 1u) {
                ev ^= ps.events[rh.ev0 + k].mask;
                gev ^= ps.events[rh.ev0 + k].gmask;
            }
        const uint32_t o = q.lo[lane] ^ q.hi[warp] ^ rh.xorc ^ ev;
        const uint32_t r0 = rh.r0, r1 = rh.r1, r2 = rh.r2, r3 = rh.r3;
        const uint32_t r01 = r0 ^ r1, r23 = r2 ^ r3; // one three-input operation per slot
        auto slot = [&](int j) {
            return o ^ ((j & 3) == 3 ? r01 : (j & 1) ? r0 : (j & 2) ? r1 : 0u) ^
                   ((j & 12) == 12 ? r23 : (j & 4) ? r2 : (j & 8) ? r3 : 0u);
        };
        V v[NA], h[NA];
        if (r == 0) {
            const TileIndex &x = ps.index[hd.load_idx];
            const uint32_t g = gev ^ x.lo[lane] ^ x.hi[warp] ^ x.c;
            const uint32_t g0 = x.r[0], g1 = x.r[1], g2 = x.r[2], g3 = x.r[3], g01 = g0 ^ g1, g23 = g2 ^ g3;
            const void *lam = bf.lam_src, *hl = bf.hl;
            auto at = [&](int j) {
                return g ^ ((j & 3) == 3 ? g01 : (j & 1) ? g0 : (j & 2) ? g1 : 0u) ^
                       ((j & 12) == 12 ? g23 : (j & 4) ? g2 : (j & 8) ? g3 : 0u);
            };
            // all loads are issued before the first is used
            if (bf.from_zero) {
#pragma unroll
                for (int j = 0; j < NA; j++) v[j] = basis_amp(at(j), V{});
            } else {
#pragma unroll
                for (int j = 0; j < NA; j++) v[j] = load_bits(lam, at(j), V{});
            }
            const uint32_t wx = bf.word ? bf.wx : 0u;
            if (BWD) {
                const void *from = bf.word ? lam : hl;
#pragma unroll
                for (int j = 0; j < NA; j++) h[j] = load_bits(from, at(j) ^ wx, V{});
            }
            if (A::kBytes == 16 && !bf.in_df) {
#pragma unroll
                for (int j = 0; j < NA; j++) {
                    if (!bf.from_zero) v[j] = from_bits(v[j]);
                    if (BWD) h[j] = from_bits(h[j]);
                }
            }
            if (BWD) {
                if (bf.word) {
#pragma unroll
                    for (int j = 0; j < NA; j++) {
                        if (bf.wq & 1u) h[j] = times_i(h[j]);
                        if ((bf.wq >> 1 ^ __popc((at(j) ^ wx) & bf.wz)) & 1u) h[j] = negate(h[j]);
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < NA; j++) {
                v[j] = A::ld(L + slot(j));
                if (BWD) h[j] = A::ld(M + slot(j));
            }
        }
        uint32_t gi = base;
        if (q.idx != 0xffffu) gi |= ps.index[q.idx].lo[lane] | ps.index[q.idx].hi[warp];
        for (int k = 0; k < (int)rh.nstages; k++) {
            const TileStage &st = ps.stages[rh.stage0 + k];
            const StageHead f(st);
            DF y[8] = {}; // Y sums by bit, then Z sums by bit
            DF x[4] = {};
            bool zbits = false;
            if (BWD && (f.table & 1)) {
                zbits = (f.zsel & ~0x0116u) == 0;
                if (zbits) walsh_bits<A, R>(v, h, y + 4);
                else walsh_all<A, R>(v, h, f.zsel, f.acc_z, row, lane);
            }
            if (f.table & 2) {
                if constexpr (A::kBytes == 8) { // two entries a read
                    const float4 *e = reinterpret_cast<const float4 *>(ps.tab + f.tab * sizeof(float2));
#pragma unroll
                    for (int j = 0; j < NA; j += 2) {
                        const float4 z = e[j / 2];
                        const float2 z0 = make_float2(z.x, z.y), z1 = make_float2(z.z, z.w);
                        phase(v[j], z0);
                        phase(v[j + 1], z1);
                        if (BWD) {
                            phase(h[j], z0);
                            phase(h[j + 1], z1);
                        }
                    }
                } else {
                    const auto *e = reinterpret_cast<const typename Form<A>::E *>(ps.tab) + f.tab;
#pragma unroll
                    for (int j = 0; j < NA; j++) {
                        const auto z = e[j];
                        phase(v[j], z);
                        if (BWD) phase(h[j], z);
                    }
                }
            }
            {
                DF(&y4)[4] = reinterpret_cast<DF(&)[4]>(y);
                step_ry<A, R, BWD, 0>(v, h, st, f.ry, y4, x);
                step_ry<A, R, BWD, 1>(v, h, st, f.ry, y4, x);
                step_ry<A, R, BWD, 2>(v, h, st, f.ry, y4, x);
                step_ry<A, R, BWD, 3>(v, h, st, f.ry, y4, x);
            }
            if (BWD) {
                if (zbits || (f.sums & 1)) {
                    int k;
                    const DF t = warp_sums<8>(y, lane, k);
                    // acc_y, then acc_zb
                    const unsigned char *ids = reinterpret_cast<const unsigned char *>(&st) + offsetof(TileStage, acc_y);
                    acc_sums<8>(row, lane, reinterpret_cast<const int16_t *>(ids)[k], t);
                }
                if (f.sums & 2) {
                    int k;
                    const DF t = warp_sums<4>(x, lane, k);
                    acc_sums<4>(row, lane, st.acc_x[k], t);
                }
            }
            if (f.special == TS_CRY) {
                const uint32_t act = (gi & st.cmask) == st.cval ? st.jact : 0u;
                DF c = {0.0f, 0.0f};
                switch (st.bit) {
                case 0: step_cry<A, R, BWD, 0>(v, h, st, act, c); break;
                case 1: step_cry<A, R, BWD, 1>(v, h, st, act, c); break;
                case 2: step_cry<A, R, BWD, 2>(v, h, st, act, c); break;
                default: step_cry<A, R, BWD, 3>(v, h, st, act, c); break;
                }
                if (BWD && st.sacc >= 0) {
                    c = warp_sum(c);
                    if (lane == 0) acc_add(row, st.sacc, c);
                }
            } else if (f.special != TS_NONE) {
                step_index<A, R, BWD>(v, h, st, ps.index[q.idx], gi, ps.tab, row, lane);
            }
        }
        if (r + 1 < nrounds) {
            // a tile of fewer threads than a warp: lanes that work alike share their
            // slots, and all have to have read them before one writes
            if (T < R + 5) __syncwarp();
#pragma unroll
            for (int j = 0; j < NA; j++) {
                A::st(L + slot(j), v[j]);
                if (BWD) A::st(M + slot(j), h[j]);
            }
        } else if (!BWD || !bf.drop) {
            if (nrounds == 1) __syncthreads(); // all of the tile read before any of it is written
            uint32_t go = base;
            for (int k = hd.ev_store0; k < hd.nev; k++)
                if (base >> ps.events[k].bit & 1u) go ^= ps.events[k].gmask;
            const TileIndex &x = ps.index[hd.store_idx];
            const uint32_t g = go ^ x.lo[lane] ^ x.hi[warp] ^ x.c;
            const uint32_t g0 = x.r[0], g1 = x.r[1], g2 = x.r[2], g3 = x.r[3], g01 = g0 ^ g1, g23 = g2 ^ g3;
            void *lam = bf.lam, *hl = bf.hl;
#pragma unroll
            for (int j = 0; j < NA; j++) {
                const uint32_t i = g ^ ((j & 3) == 3 ? g01 : (j & 1) ? g0 : (j & 2) ? g1 : 0u) ^
                                   ((j & 12) == 12 ? g23 : (j & 4) ? g2 : (j & 8) ? g3 : 0u);
                store_amp(lam, i, bf.out_df, v[j]);
                if (BWD) store_amp(hl, i, bf.out_df, h[j]);
            }
        }
        __syncthreads();
    }
}

template <class A, int R, bool BWD, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) k_tile(const __grid_constant__ Args a) {
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tile_bytes = (uint32_t)A::kBytes << a.T;
    unsigned char *L = tile_smem, *M = L + tile_bytes;
    unsigned char *prog = tile_smem + (BWD ? 2 : 1) * tile_bytes;
    float2 *acc = reinterpret_cast<float2 *>(prog + a.prog_bytes);
    float2 *row = acc + warp * a.nacc;
    for (uint32_t i = tid * 16; i < a.prog_bytes; i += blockDim.x * 16)
        *reinterpret_cast<uint4 *>(prog + i) = __ldg(reinterpret_cast<const uint4 *>(a.prog + i));
    if (BWD)
        for (int i = lane; i < a.nacc; i += 32) row[i] = make_float2(0.0f, 0.0f);
    __syncthreads();
    const Pass ps(prog);
    const Buffers bf{a.lam_src[blockIdx.y], a.lam[blockIdx.y], a.hl[blockIdx.y], a.in_df, a.out_df, false, BWD && a.drop,
                     BWD && a.words, a.wx[blockIdx.y], a.wz[blockIdx.y], a.wq[blockIdx.y]};
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) run_tile<A, R, BWD>(ps, bf, tile, a.T, L, M, row);
    if (BWD) {
        for (int i = tid; i < a.nacc; i += blockDim.x) {
            DF t = {0.0f, 0.0f};
            for (int w = 0; w < (int)blockDim.x / 32; w++) df_add(acc[w * a.nacc + i].x, acc[w * a.nacc + i].y, t.hi, t.lo);
            a.part[((size_t)blockIdx.y * a.nacc_all + ps.hd.acc0 + i) * gridDim.x + blockIdx.x] = df_result(t.hi, t.lo);
        }
    }
}

} // namespace tile
} // namespace plk
