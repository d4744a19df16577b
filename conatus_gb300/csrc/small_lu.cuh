// Solves with the LU factors of a system's small r x r capacitance matrix (one thread).
#pragma once

#include "common.cuh"

namespace cng {

// z := S^{-1} z with the small LU (getrs 'N'; 1 / u_kk on the diagonal), one thread.
template <class T>
__device__ void small_getrs(const T* a, const int* piv, T* z, int r) {
    for (int k = 0; k < r; ++k) {
        const int p = piv[k];
        if (p != k) {
            T t = z[k];
            z[k] = z[p];
            z[p] = t;
        }
    }
    for (int k = 0; k < r; ++k)
        for (int i = k + 1; i < r; ++i) z[i] = z[i] - a[k * r + i] * z[k];
    for (int k = r - 1; k >= 0; --k) {
        z[k] = z[k] * a[k * r + k];
        for (int i = 0; i < k; ++i) z[i] = z[i] - a[k * r + i] * z[k];
    }
}

}  // namespace cng
