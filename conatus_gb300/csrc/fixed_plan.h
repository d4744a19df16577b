// Host tables of the fixed-point FFT (fixed_fft.cuh): stages, twiddles and index maps of a length.
#pragma once

#include <cmath>
#include <cstdint>
#include <vector>

#include "fixed_fft.cuh"

namespace cng {

inline FxC fx_const(long double w) {            // round(w 2^62) in signed halves; |w| < 2
    const long long v = llrintl(w * 4611686018427387904.0L);
    const int l = (int)(uint32_t)(unsigned long long)v;
    return FxC{(int)((v - l) >> 32), l};
}
inline FxTw fx_twiddle(long double wr, long double wi) { return FxTw{fx_const(wr), fx_const(wi - wr), fx_const(wi + wr)}; }

struct FxTables {
    FxPlan plan;                                // its pointers are set by the owner of the tables
    std::vector<FxTw> tw;
    std::vector<uint16_t> in_pos, out_pos, k_of;
};

inline unsigned fx_recip(int d) { return d <= 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u; }

// L = 2^a 3^b 5^c <= kFxMaxLen (the caller has checked the factors)
inline FxTables fx_tables(int L) {
    const long double two_pi = 6.283185307179586476925286766559005768L;
    struct Block { int N, stride; std::vector<int> rad; };
    std::vector<Block> blocks;
    int rest = L;
    auto exponent = [&](int p) { int e = 0; while (rest % p == 0) { rest /= p; ++e; } return e; };
    const int a = exponent(2), b = exponent(3), c = exponent(5);
    if (b) {
        Block k{1, 0, {}};
        for (int i = 0; i < b / 2; ++i) k.rad.push_back(9);
        if (b % 2) k.rad.push_back(3);
        blocks.push_back(k);
    }
    if (c) blocks.push_back(Block{1, 0, std::vector<int>(c, 5)});
    if (a) {                                    // eights, and a 4, two 4s or a 2 for what is left
        Block k{1, 0, {}};
        const int fours = a % 3 == 2 ? 1 : (a % 3 == 1 && a > 1 ? 2 : 0);
        for (int i = 0; i < (a - 2 * fours) / 3; ++i) k.rad.push_back(8);
        for (int i = 0; i < fours; ++i) k.rad.push_back(4);
        if (a == 1) k.rad.push_back(2);
        blocks.push_back(k);
    }
    FxTables T;
    T.plan.L = L;
    int stride = L;
    for (auto& k : blocks) {
        for (int r : k.rad) k.N *= r;
        stride /= k.N;
        k.stride = stride;
        int n = k.N;
        for (size_t i = 0; i < k.rad.size(); ++i) {
            const int r = k.rad[i], m = n / r;
            FxStage& s = T.plan.s[T.plan.nst++];
            s.radix = r;
            s.M = m * stride;
            s.st = stride;
            s.mM = fx_recip(s.M);
            s.mst = fx_recip(s.st);
            s.tw = -1;
            if (m > 1) {                        // exp(-2 pi i j q / n)
                s.tw = (int)T.tw.size();
                for (int j = 0; j < m; ++j)
                    for (int q = 1; q < r; ++q) {
                        const long double ang = -two_pi * (long double)((long long)j * q % n) / n;
                        T.tw.push_back(fx_twiddle(cosl(ang), sinl(ang)));
                    }
            }
            n = m;
        }
    }
    if (L > 300) {
        // rescaled after the stages whose sums hold P entries: the inputs' rounding is then about 6 P / L
        // of what it was (largest entry against mean), the rescaling adds one rounding per L / P entries
        double least = 0;
        long long P = 1;
        for (int i = 0; i + 1 < T.plan.nst; ++i) {
            P *= T.plan.s[i].radix;
            const double err = 36.0 * P * P / L + (double)L / P;
            if (i > 0 && err >= least) continue;
            least = err;
            T.plan.shift_at = i + 1;
            T.plan.shift_log = 0;
            while ((1 << T.plan.shift_log) < 1.5 * P) ++T.plan.shift_log;
        }
    }
    T.in_pos.resize(L);
    T.out_pos.resize(L);
    T.k_of.resize(L);
    for (int n = 0; n < L; ++n) {
        int pin = 0, pout = 0;
        for (const auto& k : blocks) {
            int inv = 1;                        // (L / N)^-1 mod N
            while ((long long)inv * (L / k.N) % k.N != 1 % k.N) ++inv;
            pin += (int)((long long)n * inv % k.N) * k.stride;
            int q = n % k.N, size = k.N, at = 0;    // output digits: first stage's least significant
            for (int r : k.rad) {
                size /= r;
                at += (q % r) * size;
                q /= r;
            }
            pout += at * k.stride;
        }
        T.in_pos[n] = (uint16_t)pin;
        T.out_pos[n] = (uint16_t)pout;
        T.k_of[pout] = (uint16_t)n;
    }
    return T;
}

}  // namespace cng
