// Derivative expansion fused into the load of a backward transform (fields that differ only by a
// derivative along the transform's axis share the transforms before it): output group og of the
// batch reads input group src[og] and multiplies each value by (i k_j)^ord[og], k_j the wavenumber
// of its index j along the axis, from a table [order - 1][nidx] rounded to R on the host. Outer row
// o = (c nout + og) per + r reads row (c nin + src[og]) per + r.
#pragma once

#include "fft.cuh"

namespace cng {

template <class R>
struct Expand {
    int nout = 0;                 // 0: no expansion (row o reads row o)
    int nin = 0, per = 1, nidx = 0;
    const int* src = nullptr;
    const int* ord = nullptr;
    const c2<R>* tab = nullptr;
};

// the source row of outer row o and its factor table (nullptr: no derivative)
template <class R>
__device__ __forceinline__ long long expand_row(const Expand<R>& ex, long long o, const c2<R>** wt) {
    *wt = nullptr;
    if (ex.nout == 0) return o;
    const long long g = o / ex.per;
    const long long r = o - g * ex.per;
    const long long c = g / ex.nout;
    const int og = (int)(g - c * ex.nout);
    const int od = ex.ord[og];
    if (od > 0) *wt = ex.tab + (size_t)(od - 1) * ex.nidx;
    return (c * ex.nin + ex.src[og]) * ex.per + r;
}

// w v with w = (i k)^o (the product of the separate expansion pass)
template <class R>
__device__ __forceinline__ c2<R> ikmul(c2<R> w, c2<R> v) {
    return mk<R>(w.x * v.x - w.y * v.y, w.x * v.y + w.y * v.x);
}

}  // namespace cng
