// Real form of complex tau systems. In a Fourier-Chebyshev discretization a factor i comes with every
// odd Fourier derivative, so the matrices are real up to powers of i: A_kj = i^{p_k - q_j} R_kj with R
// real, p, q in {0, 1}. Then A x = b is R x' = b' with b'_k = i^{-p_k} b_k and x_j = i^{q_j} x'_j, exact
// exchanges and sign changes, and a complex product takes two fused multiply-adds instead of four
// (the other two add exact zeros, so the results are the same bits). The factors of A are the ones of
// R with the same phases: L entries carry p_row - p_pivot, U entries p_row - q_col, W columns
// q_row - p_border, and the pivot search compares the same magnitudes.
#pragma once

#include <vector>

#include "common.cuh"

namespace cng {

// the real number r of v = i^dp r (dp in {-1, 0, 1}); `bad` is set where v is not of that form
__device__ __forceinline__ double real_part_of(double v, int, int&) { return v; }
__device__ __forceinline__ double real_part_of(zd v, int dp, int& bad) {
    const bool imag = dp != 0;
    if ((imag ? v.re : v.im) != 0.0) bad = 1;
    return imag ? (dp > 0 ? v.im : -v.im) : v.re;
}
// -v on the sign bit: an FP64 negation is an instruction of the FP64 unit
__device__ __forceinline__ double flip(double v) { return __hiloint2double(__double2hiint(v) ^ (int)0x80000000, __double2loint(v)); }
__device__ __forceinline__ float flip(float v) { return -v; }
// i^-p b and i^q x
template <class T>
__device__ __forceinline__ T phase_in(T b, int p) { return p ? T(b.im, flip(b.re)) : b; }

// Row and column phases of the assembled systems (band `ab` and border rows `vt`, before the
// factorization), found on every (batch / 256)-th of them; false where there are none. What is built from
// the factors has to check every value and every row's phase of every system against them.
bool find_phases(const zd* ab, const zd* vt, int batch, int n, int r, int kv, int ldab, cudaStream_t st,
                 std::vector<unsigned char>& row, std::vector<unsigned char>& col);

}  // namespace cng
