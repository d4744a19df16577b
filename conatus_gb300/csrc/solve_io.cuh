// Input/output adapters of the solve kernels: plain in-place, mapped (int64 gather/scatter maps),
// split (complex system with real data: b = re[rows_c] + i re[rows_s]) and mixed (complex128 data,
// FP32 factors).
#pragma once

#include "common.cuh"

namespace cng {

enum IoKind { IO_PLAIN = 0, IO_MAPPED = 1, IO_SPLIT = 2, IO_MIXED = 3 };

struct SolveIo {
    const void* rhs;
    void* x;
    const long long* rows;
    const long long* cols;
    const long long* rows_s;
    const long long* cols_s;
    int accumulate = 0;
    void* xT = nullptr;            // IO_MIXED: x also written row-major over the systems, [n][batch]
};

template <class T, int IO>
__device__ inline T io_load(const SolveIo& io, int sys, int n, int i) {
    const size_t k = (size_t)sys * n + i;
    if constexpr (IO == IO_PLAIN) {
        return static_cast<const T*>(io.rhs)[k];
    } else if constexpr (IO == IO_MAPPED) {
        const T* rhs = static_cast<const T*>(io.rhs);
        return rhs[io.rows ? io.rows[k] : (long long)k];
    } else {
        const double* re = static_cast<const double*>(io.rhs);
        return T(zd(re[io.rows[k]], re[io.rows_s[k]]));
    }
}

template <class T, int IO>
__device__ inline void io_store(const SolveIo& io, int sys, int n, int i, T v) {
    const size_t k = (size_t)sys * n + i;
    if constexpr (IO == IO_PLAIN) {
        static_cast<T*>(io.x)[k] = v;
    } else if constexpr (IO == IO_MAPPED) {
        static_cast<T*>(io.x)[io.cols ? io.cols[k] : (long long)k] = v;
    } else {
        double* x = static_cast<double*>(io.x);
        const zd z = *reinterpret_cast<const zd*>(&v);
        x[io.cols[k]] = z.re;
        x[io.cols_s[k]] = z.im;
    }
}

}  // namespace cng
