// 64-bit fixed-point batched FFT core of the FP64 transforms.
//
// The GB300 issues FP64 at 1/64 of the FP32 rate (measured: 1.7 of 2 fused multiply-adds per clock
// and SM), while it does 58 64-bit integer additions and 4.3 64 x 64-bit fixed-point products per
// clock and SM. An FFT is mostly additions, and each of its outputs is a sum over one column, so its
// FP64 error is absolute in the column's norm: block floating point in 64-bit integers with one
// exponent per column loses nothing against the column's norm. A column is scaled so that the sum of its
// entries' magnitudes, which bounds every intermediate sum, is below 2^61: its largest entries keep up to 61
// bits (about 53 in flat columns of 288 points, the least), the smaller ones fewer by their size. Measured
// against 128-bit transforms, the error relative to the norm is below the FP64 transforms' for flat and
// for decaying spectra (tests/test_fixed_transforms*.py).
//
// Products being the expensive part (13 additions each), the transforms are built for few of them:
// L = 2^a 3^b 5^c is split by the prime-factor map (Good 1958, Thomas 1963) into blocks with no
// twiddles between them, each block runs in-place decimation-in-frequency stages of radix 2, 3, 4,
// 5, 8 and 9, the radix-3, -5 and -9 butterflies in the few-multiplication forms that follow from
// their cyclic convolutions (Rader 1968, Winograd 1978; radix 9: 8 real constants per complex
// butterfly), and a twiddle takes three products (wr (x + y) and two corrections). L = 288 takes
// about 1250 products per complex transform where the direct mixed radix takes 3700.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace cng {

#define FX_HD __host__ __device__ __forceinline__

using fx = long long;
struct alignas(16) fx2 { fx x, y; };

// A constant in Q62, split as (h + l 2^-32) 2^-30 with signed halves.
struct FxC { int h, l; };
// A twiddle w = wr + i wi as (wr, wi - wr, wi + wr).
struct FxTw { FxC r, d, s; };

FX_HD int fx_hi(fx a) { return (int)((unsigned long long)(a + 0x80000000LL) >> 32); }   // a = hi 2^32 + (int)a
// (2^32 h + c) 2^-30 rounded, c already holding the rounding constant 2^29
FX_HD fx fx_join(fx h, fx c) { return (fx)((unsigned long long)h << 2) + (c >> 30); }

// a w, |w| < 2: three 32 x 32 -> 64 products (the fourth is below the last bit)
FX_HD fx fx_mul(fx a, FxC w) {
    const int h = fx_hi(a), l = (int)a;
    const fx c = (fx)h * w.l + (fx)l * w.h + (1LL << 29);
    return fx_join((fx)h * w.h, c);
}
// a u + b v, |u|, |v| <= 1
FX_HD fx fx_mul2(fx a, FxC u, fx b, FxC v) {
    const int ah = fx_hi(a), al = (int)a, bh = fx_hi(b), bl = (int)b;
    const fx c = (fx)ah * u.l + (fx)al * u.h + (fx)bh * v.l + (fx)bl * v.h + (1LL << 29);
    return fx_join((fx)ah * u.h + (fx)bh * v.h, c);
}
FX_HD fx2 fx_add(fx2 a, fx2 b) { return {a.x + b.x, a.y + b.y}; }
FX_HD fx2 fx_sub(fx2 a, fx2 b) { return {a.x - b.x, a.y - b.y}; }
FX_HD fx2 fx_mulr(fx2 a, FxC w) { return {fx_mul(a.x, w), fx_mul(a.y, w)}; }
// a w
FX_HD fx2 fx_cmul(fx2 a, const FxTw& w) {
    const fx t = fx_mul(a.x + a.y, w.r);
    return {t - fx_mul(a.y, w.s), t + fx_mul(a.x, w.d)};
}
// a - i b and a + i b
FX_HD fx2 fx_sub_i(fx2 a, fx2 b) { return {a.x + b.y, a.y - b.x}; }
FX_HD fx2 fx_add_i(fx2 a, fx2 b) { return {a.x - b.y, a.y + b.x}; }

// ---- butterflies: forward DFTs (exp(-2 pi i nk / R)) in place -----------------------------------
// the constants are cos and sin of multiples of 2 pi / R (and their combinations) in Q62
FX_HD void fx_dft2(fx2* v) {
    const fx2 a = v[0], b = v[1];
    v[0] = fx_add(a, b);
    v[1] = fx_sub(a, b);
}
FX_HD void fx_dft4(fx2& v0, fx2& v1, fx2& v2, fx2& v3) {
    const fx2 a0 = fx_add(v0, v2), a1 = fx_sub(v0, v2), b0 = fx_add(v1, v3), b1 = fx_sub(v1, v3);
    v0 = fx_add(a0, b0);
    v2 = fx_sub(a0, b0);
    v1 = fx_sub_i(a1, b1);
    v3 = fx_add_i(a1, b1);
}
FX_HD void fx_dft8(fx2* v) {
    constexpr FxC h = {759250125, -25716447};                       // sqrt(1/2)
    fx_dft4(v[0], v[2], v[4], v[6]);
    fx_dft4(v[1], v[3], v[5], v[7]);
    // odd outputs o_k times exp(-i pi k / 4)
    const fx2 o1 = {fx_mul(v[3].x + v[3].y, h), fx_mul(v[3].y - v[3].x, h)};
    const fx2 o3 = {fx_mul(v[7].y - v[7].x, h), fx_mul(v[7].x + v[7].y, h)};     // (x, -y) of the product
    const fx2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o2 = v[5];
    v[0] = fx_add(e0, o0);
    v[4] = fx_sub(e0, o0);
    v[1] = fx_add(e1, o1);
    v[5] = fx_sub(e1, o1);
    v[2] = fx_sub_i(e2, o2);
    v[6] = fx_add_i(e2, o2);
    v[3] = {e3.x + o3.x, e3.y - o3.y};
    v[7] = {e3.x - o3.x, e3.y + o3.y};
}
FX_HD void fx_dft3(fx2* v) {
    constexpr FxC s = {929887697, -1332128537};                     // sin 120
    const fx2 t1 = fx_add(v[1], v[2]), t2 = fx_mulr(fx_sub(v[1], v[2]), s);
    const fx2 m = {v[0].x - (t1.x >> 1), v[0].y - (t1.y >> 1)};
    v[0] = fx_add(v[0], t1);
    v[1] = fx_sub_i(m, t2);
    v[2] = fx_add_i(m, t2);
}
FX_HD void fx_dft5(fx2* v) {
    constexpr FxC r5 = {600239927, 803819395};                      // sqrt(5)/4
    constexpr FxC s2 = {631129609, -357254181};                     // sin 144
    constexpr FxC sd = {390059550, -1644870943};                    // sin 72 - sin 144
    constexpr FxC sp = {1652318767, 1935587992};                    // sin 72 + sin 144
    const fx2 p1 = fx_add(v[1], v[4]), m1 = fx_sub(v[1], v[4]), p2 = fx_add(v[2], v[3]), m2 = fx_sub(v[2], v[3]);
    const fx2 t = fx_add(p1, p2), d = fx_mulr(fx_sub(p1, p2), r5);
    const fx2 u = {v[0].x - (t.x >> 2), v[0].y - (t.y >> 2)};
    const fx2 a1 = fx_add(u, d), a2 = fx_sub(u, d);
    const fx2 q = fx_mulr(fx_add(m1, m2), s2);
    const fx2 b1 = fx_add(q, fx_mulr(m1, sd)), b2 = fx_sub(q, fx_mulr(m2, sp));
    v[0] = fx_add(v[0], t);
    v[1] = fx_sub_i(a1, b1);
    v[4] = fx_add_i(a1, b1);
    v[2] = fx_sub_i(a2, b2);
    v[3] = fx_add_i(a2, b2);
}
// cos and sin sums over n = 1, 2, 4 are length-3 cyclic convolutions (2 generates the units mod 9):
// with cos 40 + cos 80 + cos 160 = 0 and sin 80 = sin 40 + sin 160, three products each
FX_HD void fx_dft9(fx2* v) {
    constexpr FxC ca = {186453311, 96060625};                       // cos 80
    constexpr FxC cb = {636080647, -1729712749};                    // cos 40 - cos 80
    constexpr FxC cc = {1195440580, -1441530873};                   // cos 40 + 2 cos 80
    constexpr FxC sa = {690187940, 2016164183};                     // sin 40
    constexpr FxC sb = {367241333, -1978927779};                    // sin 160
    constexpr FxC sc = {1057429273, 37236404};                      // sin 80
    constexpr FxC s3 = {929887697, -1332128537};                    // sin 120
    const fx2 p1 = fx_add(v[1], v[8]), p2 = fx_add(v[2], v[7]), p3 = fx_add(v[3], v[6]), p4 = fx_add(v[4], v[5]);
    const fx2 m1 = fx_sub(v[1], v[8]), m2 = fx_sub(v[2], v[7]), m3 = fx_sub(v[3], v[6]), m4 = fx_sub(v[4], v[5]);
    const fx2 z = v[0], t = fx_add(fx_add(p1, p2), p4);
    const fx2 w = {z.x - (p3.x >> 1), z.y - (p3.y >> 1)}, z3 = fx_add(z, p3);
    const fx2 a = fx_sub(p1, p4), b = fx_sub(p2, p4);
    const fx2 q = fx_mulr(fx_add(a, b), ca);
    const fx2 c1 = fx_add(q, fx_mulr(a, cb)), c2 = fx_sub(q, fx_mulr(b, cc));
    const fx2 e = fx_add(m1, m2), f = fx_add(m2, m4);
    const fx2 g = fx_mulr(fx_sub(e, f), sa), h = fx_mulr(e, sb), k = fx_mulr(f, sc), n3 = fx_mulr(m3, s3);
    const fx2 S3 = fx_mulr(fx_add(fx_sub(m1, m2), m4), s3);
    const fx2 C1 = fx_add(w, c1), C2 = fx_add(w, c2), C4 = fx_sub(w, fx_add(c1, c2));
    const fx2 S1 = fx_add(fx_add(g, k), n3), S2 = fx_sub(fx_add(g, h), n3), S4 = fx_add(fx_sub(h, k), n3);
    const fx2 C3 = {z3.x - (t.x >> 1), z3.y - (t.y >> 1)};
    v[0] = fx_add(z3, t);
    v[1] = fx_sub_i(C1, S1);
    v[8] = fx_add_i(C1, S1);
    v[2] = fx_sub_i(C2, S2);
    v[7] = fx_add_i(C2, S2);
    v[3] = fx_sub_i(C3, S3);
    v[6] = fx_add_i(C3, S3);
    v[4] = fx_sub_i(C4, S4);
    v[5] = fx_add_i(C4, S4);
}
template <int RAD>
FX_HD void fx_dft(fx2* v) {
    if constexpr (RAD == 2) fx_dft2(v);
    else if constexpr (RAD == 3) fx_dft3(v);
    else if constexpr (RAD == 4) fx_dft4(v[0], v[1], v[2], v[3]);
    else if constexpr (RAD == 5) fx_dft5(v);
    else if constexpr (RAD == 8) fx_dft8(v);
    else fx_dft9(v);
}

// ---- plan ---------------------------------------------------------------------------------------
// Position p of the in-place array: mixed radix over the prime-power blocks. Entry n of the input
// goes to in_pos[n]; after the stages output k is at out_pos[k] (k_of is its inverse).
constexpr int kFxMaxStages = 10;
constexpr int kFxMaxLen = 16384;
struct FxStage {
    int radix, M, st, tw;           // stride M between a butterfly's elements, st of its block; twiddles at
                                    // tw + j (radix - 1) + q - 1, or tw < 0: none (the block's last stage)
    unsigned mM, mst;               // multiply-high reciprocals of M and st
};
struct FxPlan {
    int L = 0, nst = 0;
    int shift_at = 0, shift_log = 0;            // long columns: the stage whose inputs are rescaled (fx_base), 0: none
    FxStage s[kFxMaxStages] = {};
    const FxTw* tw = nullptr;
    const uint16_t* in_pos = nullptr;
    const uint16_t* out_pos = nullptr;
    const uint16_t* k_of = nullptr;
};
FX_HD unsigned fx_div(unsigned e, unsigned d, unsigned m) {         // e / d, m = ceil(2^32 / d), e < 2^14 * 64
#ifdef __CUDA_ARCH__
    return d <= 1 ? e : __umulhi(e, m);
#else
    (void)m;
    return e / d;
#endif
}

// (v + half) >> g
FX_HD fx2 fx_shift(fx2 v, int g) {
    const fx half = (1LL << g) >> 1;
    return {(v.x + half) >> g, (v.y + half) >> g};
}

// One stage over the columns c < C of z[p CS + c] (C = 1 << lc): the butterflies idx = tid, tid + nt, ...
// `out(p, c, v)` takes the results; `shift(c)` is the rescaling of the stage's inputs in bits.
template <int RAD, class Out, class Shift>
FX_HD void fx_stage(fx2* z, const FxPlan& pl, const FxStage& s, int lc, int CS, int tid, int nt, Out&& out, Shift&& shift) {
    const int total = (pl.L / RAD) << lc;
    for (int idx = tid; idx < total; idx += nt) {
        const int c = idx & ((1 << lc) - 1);
        const unsigned b = (unsigned)idx >> lc;
        const unsigned blk = fx_div(b, s.M, s.mM), rem = b - blk * s.M;
        const int p0 = (int)(blk * RAD * s.M + rem);
        fx2* zp = z + (size_t)p0 * CS + c;
        fx2 v[RAD];
#pragma unroll
        for (int t = 0; t < RAD; ++t) v[t] = zp[t * s.M * CS];
        if (const int g = shift(c)) {
#pragma unroll
            for (int t = 0; t < RAD; ++t) v[t] = fx_shift(v[t], g);
        }
        fx_dft<RAD>(v);
        if (s.tw >= 0) {
            const unsigned j = fx_div(rem, s.st, s.mst);
            if (j) {
                const FxTw* w = pl.tw + s.tw + j * (RAD - 1);
#pragma unroll
                for (int q = 1; q < RAD; ++q) v[q] = fx_cmul(v[q], w[q - 1]);
            }
        }
#pragma unroll
        for (int t = 0; t < RAD; ++t) out(p0 + t * s.M, c, v[t]);
    }
}
template <class Out, class Shift>
FX_HD void fx_stage_any(fx2* z, const FxPlan& pl, const FxStage& s, int lc, int CS, int tid, int nt, Out&& out, Shift&& shift) {
    switch (s.radix) {
        case 2: fx_stage<2>(z, pl, s, lc, CS, tid, nt, out, shift); break;
        case 3: fx_stage<3>(z, pl, s, lc, CS, tid, nt, out, shift); break;
        case 4: fx_stage<4>(z, pl, s, lc, CS, tid, nt, out, shift); break;
        case 5: fx_stage<5>(z, pl, s, lc, CS, tid, nt, out, shift); break;
        case 8: fx_stage<8>(z, pl, s, lc, CS, tid, nt, out, shift); break;
        default: fx_stage<9>(z, pl, s, lc, CS, tid, nt, out, shift); break;
    }
}

// ---- conversion ---------------------------------------------------------------------------------
// A column's exponent e (largest biased exponent, at least 1) and the sum T of (mantissa >> (36 + e -
// own exponent)) + 1 over its reals bound the sum of magnitudes by T 2^(e - 1039); lg bits of T
// (at least 17) and x further bits of headroom put it below 2^61: fixed = value 2^(1086 - base) with
// base = lg + e + x - 14.
//
// That scale wastes the bits of the early stages, whose sums are short: in a long column of flat
// magnitude the rounding of the inputs, summed over L of them, would exceed the FP64 transforms' error
// (measured from L of about 350). So the columns of long plans start up to 8 bits finer, as far as
// the stages before `shift_at` (sums of P entries: shift_log bits) allow, and are rescaled there.
struct FxScale { int base, shift; };            // fixed = value 2^(1086 - base) until `shift` bits are dropped
FX_HD FxScale fx_base(const FxPlan& pl, int emax, unsigned T, int x) {
#ifdef __CUDA_ARCH__
    const int bits = 32 - __clz((int)T);
#else
    const int bits = T ? 32 - __builtin_clz(T) : 0;
#endif
    FxScale f;
    const int base = (bits > 17 ? bits : 17) + emax + x - 14;
    f.base = base;
    if (pl.shift_at) {
        int b = emax + x + 3 + pl.shift_log;
        b = b > base - 8 ? b : base - 8;
        f.base = b < base ? b : base;
    }
    f.shift = base - f.base;
    return f;
}
FX_HD int fx_hiword(double d) {
#ifdef __CUDA_ARCH__
    return __double2hiint(d);
#else
    long long b;
    __builtin_memcpy(&b, &d, 8);
    return (int)(b >> 32);
#endif
}
FX_HD unsigned fx_loword(double d) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(d);
#else
    long long b;
    __builtin_memcpy(&b, &d, 8);
    return (unsigned)b;
#endif
}
FX_HD unsigned fx_weight(double d, int emax) {
    const int hi = fx_hiword(d);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned m = ((unsigned)hi & 0xfffffu) | (e ? 0x100000u : 0u);
    const int sh = emax - (e ? e : 1);
    return ((m >> 4) >> (sh > 31 ? 31 : sh)) + 1;
}
FX_HD fx fx_from(double d, int base) {
    const int hi = fx_hiword(d);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned m = ((unsigned)hi & 0xfffffu) | (e ? 0x100000u : 0u);
    fx v = (fx)(((unsigned long long)m << 42) | ((unsigned long long)fx_loword(d) << 10));
    if (hi < 0) v = -v;
    int s = base - 2 - (e ? e : 1);               // value 2^(1086 - base): the 10-bit pre-shift, then one
    s = s > 62 ? 62 : s;                          // bit less than the whole shift, and the rounding
    return ((v >> s) + 1) >> 1;
}
// v 2^(base - 1086) rounded to double; 66 <= base <= 2046 keeps the exponent in range (fx_plain)
FX_HD bool fx_plain(int base) { return base >= 66 && base <= 2046; }
FX_HD double fx_to(fx v, int base) {
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
#ifdef __CUDA_ARCH__
    const unsigned h = (unsigned)(a >> 32);
    int z = __clz((int)h);
    if (h == 0) z = 32 + __clz((int)(unsigned)a);
#else
    const int z = a ? __builtin_clzll(a) : 64;
#endif
    const unsigned long long n = ((a << (z - 1)) + 0x200ull) >> 10;       // 53 bits, the top one at 52
    unsigned long long b = ((unsigned long long)(unsigned)(base - z - 1) << 52) + n;
    b |= (unsigned long long)v & 0x8000000000000000ull;
    if (a == 0) b = 0;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double d;
    __builtin_memcpy(&d, &b, 8);
    return d;
#endif
}

}  // namespace cng
