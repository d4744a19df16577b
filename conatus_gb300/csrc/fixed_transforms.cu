// The FP64 transforms of the spectral pipeline in 64-bit fixed point (fixed_fft.cuh): Chebyshev
// columns, complex and real Fourier axes. A block loads C columns once from global memory, finds each
// column's scale, converts, runs the in-place stages in shared memory and stores the results as
// doubles, the last stage straight from registers where its outputs are what is stored.
//
// What bounds them: 32 x 32 -> 64-bit products (12 per clock and SM) and the integer additions and
// conversions beside them; the FP64 transforms they replace kept the FP64 pipe 85 % busy. Measured on the
// channel 192 x 129 x 192 (x backward: 12 fields of 57600 columns, 96 modes -> 288 points, 2.65 GB):
// 5.5 -> 1.57 ms; the whole right-hand side 14.7 -> 5.0 ms (4.76 with the later products).
//
// A column that holds a NaN or an infinity comes out as NaN throughout (a transform mixes every entry
// into every output); zeros, denormals and the largest exponents are kept.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <mutex>

#include "conatus_gb300.h"
#include "fixed_plan.h"
#include "fixed_transforms.cuh"

namespace cng {

constexpr int kFxThreads = 256;                  // most threads of a block
constexpr int kFxCols = 16;                      // most columns of a block
constexpr size_t kFxSmem = 200 * 1024;

struct FxChebArgs {
    const double2* in;
    double2* out;
    long long ncols;
    int N, lc;                                   // columns per block: 1 << lc
    FxPlan plan;
    const FxTw* bq;                              // backward: (-1)^k / 2 exp(i pi k / 2M)
    const FxC* fq;                               // forward: the post-twiddle's (x, y), scaled
    int fshift;                                  // forward: exponent of that scale
};
struct FxAxisArgs {
    const void* in;
    void* out;
    long long outer;
    int inner, nc, lc;
    FxPlan plan;
    FxC scale;                                   // forward: 1/L (real: 1/2L) times 2^shift, in [1/2, 1)
    int shift;
    int wide;                                    // real backward: every pair of the output is 16-byte aligned
    Expand<double> ex;
};

// v 2^(base - 1086) outside the exponent range of fx_to, and the columns with non-finite input
static __device__ __noinline__ double fx_to_any(fx v, int base, bool bad) {
    if (bad) return __longlong_as_double(0x7ff8000000000000LL);
    const int e = base - 1086, h = e / 2;
    return ldexp(ldexp((double)v, h), e - h);
}
struct FxCol {
    int base, shift;
    bool bad;
    __device__ __forceinline__ double to(fx v, int drop) const {
        const int b = base + shift - drop;
        return !bad && fx_plain(b) ? fx_to(v, b) : fx_to_any(v, b, bad);
    }
};
// of a column's largest entry: the exponent from bit 20 on, and 0 for a column of zeros alone
__device__ __forceinline__ int fx_magnitude(double d) { return (fx_hiword(d) & 0x7fffffff) | (fx_loword(d) ? 1 : 0); }
// its exponent field. Zeros take that of 1, which keeps them (and fields that are not excited, or modes
// whose derivative is zero) off the slow way back for the ends of the range: a right-hand side of a zero
// state 9.5 ms on the channel 192 x 129 x 192 without this, 4.9 with it (a random state 4.8)
__device__ __forceinline__ int fx_column(int magnitude) { return magnitude ? max(magnitude >> 20, 1) : 1023; }

template <class Out, class Shift>
__device__ __forceinline__ void fx_stages(fx2* z, const FxPlan& pl, int n, int lc, int CS, Out&& out, Shift&& shift) {
    for (int s = 0; s < n; ++s) {
        fx_stage_any(z, pl, pl.s[s], lc, CS, threadIdx.x, blockDim.x, out,
                     [&](int c) { return s && s == pl.shift_at ? shift(c) : 0; });
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// Fourier transforms along a strided axis: data [outer][len][inner], the conventions of
// cng_fft_axis and cng_rfft_axis. REAL: a column is two adjacent inner columns a + i b (an odd last
// one is paired with zero). The columns of a block are its fastest thread index: loads and stores are
// contiguous across them, and every access to z[p][c] is free of bank conflicts.
//
// Inverse transforms run as forward ones on (y, x): the exchange costs nothing at the load and store.
template <bool REAL, bool FWD>
__device__ __forceinline__ void fx_axis_body(unsigned bid, const FxAxisArgs& a) {
    extern __shared__ __align__(16) unsigned char fx_sm[];
    __shared__ int s_e[kFxCols];
    __shared__ unsigned s_t[kFxCols];
    fx2* z = reinterpret_cast<fx2*>(fx_sm);
    const FxPlan& pl = a.plan;
    const int lc = a.lc, C = 1 << lc, L = pl.L;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, c = tid & (C - 1);
    const int cols = REAL ? (a.inner + 1) / 2 : a.inner;
    const unsigned chunks = (unsigned)((cols + C - 1) >> lc);
    const long long o = bid / chunks;
    const int col = (int)(bid - o * chunks) * C + c;              // this thread's column (every item of it)
    const bool valid = col < cols;
    if (tid < C) {
        s_e[tid] = 0;
        s_t[tid] = 0;
    }
    // item e >> lc of column c: entry k of the compact spectrum, or grid point j
    constexpr int NV = REAL && !FWD ? 4 : 2;                      // doubles of an item
    constexpr int H = NV == 4 ? 4 : 8;                            // items held in registers
    const int items = (FWD ? L : a.nc) << lc;
    const double2* wt = nullptr;
    const long long row = FWD ? o : expand_row<double>(a.ex, o, &wt);
    const bool pair = !REAL || 2 * col + 1 < a.inner;
    auto load = [&](int e, double* d) {
        const int k = e >> lc;
#pragma unroll
        for (int q = 0; q < NV; ++q) d[q] = 0.0;
        if (!valid || e >= items) return;
        if constexpr (REAL && FWD) {
            const double* s = static_cast<const double*>(a.in) + (row * L + k) * a.inner + 2 * col;
            d[0] = s[0];
            if (pair) d[1] = s[1];
        } else {
            if (!REAL && !FWD && k == a.nc / 2) return;           // the Nyquist entry is not used
            const double2* s = static_cast<const double2*>(a.in) +
                               (row * (FWD ? L : a.nc) + k) * a.inner + (REAL ? 2 * col : col);
            const double2 v = s[0];
            d[0] = v.x;
            d[1] = v.y;
            if constexpr (NV == 4) {
                if (pair) {
                    const double2 w = s[1];
                    d[2] = w.x;
                    d[3] = w.y;
                }
            }
            if (!FWD && wt) {                                     // times (i k)^o, real or imaginary
                const double2 w = wt[k];
#pragma unroll
                for (int q = 0; q < NV; q += 2) {
                    const double x = d[q], y = d[q + 1];
                    d[q] = w.y == 0.0 ? w.x * x : -w.y * y;
                    d[q + 1] = w.y == 0.0 ? w.x * y : w.y * x;
                }
            }
        }
    };
    double held[H][NV];
    const bool hold = items <= H * nt;
    int em = 0;
    if (hold) {
#pragma unroll
        for (int u = 0; u < H; ++u) load(tid + u * nt, held[u]);
#pragma unroll
        for (int u = 0; u < H; ++u)
#pragma unroll
            for (int q = 0; q < NV; ++q) em = max(em, fx_magnitude(held[u][q]));
    } else {
        for (int e = tid; e < items; e += nt) {
            load(e, held[0]);
#pragma unroll
            for (int q = 0; q < NV; ++q) em = max(em, fx_magnitude(held[0][q]));
        }
    }
    __syncthreads();
    for (int m = C; m < 32; m <<= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, m));
    if (lane < C) atomicMax(&s_e[c], em);
    __syncthreads();
    em = fx_column(s_e[c]);
    FxCol fc;
    fc.bad = em == 0x7ff;
    unsigned T = 0;
    if (hold) {
#pragma unroll
        for (int u = 0; u < H; ++u)
            if (tid + u * nt < items)
#pragma unroll
                for (int q = 0; q < NV; ++q) T += fx_weight(held[u][q], em);
    } else {
        for (int e = tid; e < items; e += nt) {
            load(e, held[0]);
#pragma unroll
            for (int q = 0; q < NV; ++q) T += fx_weight(held[0][q], em);
        }
    }
    for (int m = C; m < 32; m <<= 1) T += __shfl_xor_sync(0xffffffffu, T, m);
    if (lane < C) atomicAdd(&s_t[c], T);
    __syncthreads();
    {   // the real backward transform uses each entry twice (modes k and L - k)
        const FxScale f = fx_base(pl, em, s_t[c], NV == 4 ? 1 : 0);
        fc.base = f.base;
        fc.shift = f.shift;
    }
    auto put = [&](int n, fx x, fx y) { z[((size_t)pl.in_pos[n] << lc) + c] = FWD ? fx2{x, y} : fx2{y, x}; };
    auto convert = [&](int e, const double* d) {
        if (e >= items) return;
        const int k = e >> lc;
        fx f[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) f[q] = fc.bad ? 0 : fx_from(d[q], fc.base);
        if constexpr (NV == 4) {                                  // A + i B at k, conj(A) + i conj(B) at L - k
            put(k, f[0] - f[3], f[1] + f[2]);
            if (k) put(L - k, f[0] + f[3], f[2] - f[1]);
        } else if constexpr (FWD) {
            put(k, f[0], f[1]);
        } else {
            if (k != a.nc / 2) put(k < a.nc / 2 ? k : L - a.nc + k, f[0], f[1]);
        }
    };
    if (hold) {
#pragma unroll
        for (int u = 0; u < H; ++u) convert(tid + u * nt, held[u]);
    } else {
        for (int e = tid; e < items; e += nt) {
            load(e, held[0]);
            convert(e, held[0]);
        }
    }
    if constexpr (!FWD) {                                         // the padding
        const int n0 = REAL ? a.nc : a.nc / 2, n1 = min(L, L - a.nc + (REAL ? 0 : a.nc / 2) + 1);
        for (int e = tid + (n0 << lc); e < n1 << lc; e += nt) put(e >> lc, 0, 0);
    }
    __syncthreads();
    auto smem = [&](int p, int cc, fx2 v) { z[((size_t)p << lc) + cc] = v; };
    auto shift = [&](int) { return fc.shift; };
    if constexpr (REAL && FWD) {
        fx_stages(z, pl, pl.nst, lc, C, smem, shift);
        double2* dst = static_cast<double2*>(a.out) + o * (long long)a.nc * a.inner + 2 * col;
        if (!valid) return;
        for (int e = tid; e < a.nc << lc; e += nt) {
            const int k = e >> lc;
            const fx2 p = z[((size_t)pl.out_pos[k] << lc) + c], q = z[((size_t)pl.out_pos[k ? L - k : 0] << lc) + c];
            // (p + conj q) / 2L and (p - conj q) / 2iL
            const fx ax = fx_mul(p.x + q.x, a.scale), ay = fx_mul(p.y - q.y, a.scale);
            const fx bx = fx_mul(p.y + q.y, a.scale), by = fx_mul(q.x - p.x, a.scale);
            double2* d = dst + (long long)k * a.inner;
            d[0] = make_double2(fc.to(ax, a.shift), fc.to(ay, a.shift));
            if (pair) d[1] = make_double2(fc.to(bx, a.shift), fc.to(by, a.shift));
        }
    } else {
        auto store = [&](int p, int, fx2 v) {
            if (!valid) return;
            const int k = pl.k_of[p];
            if constexpr (FWD) {
                const int K = a.nc / 2;
                if (k >= K && k <= L - K) return;
                const int slot = k < K ? k : a.nc - (L - k);
                static_cast<double2*>(a.out)[(o * a.nc + slot) * (long long)a.inner + col] =
                    make_double2(fc.to(fx_mul(v.x, a.scale), a.shift), fc.to(fx_mul(v.y, a.scale), a.shift));
            } else if constexpr (REAL) {
                double* d = static_cast<double*>(a.out) + (o * L + k) * (long long)a.inner + 2 * col;
                const double x = fc.to(v.y, 0), y = fc.to(v.x, 0);
                if (a.wide) {
                    *reinterpret_cast<double2*>(d) = make_double2(x, y);
                } else {
                    d[0] = x;
                    if (pair) d[1] = y;
                }
            } else {
                static_cast<double2*>(a.out)[(o * L + k) * (long long)a.inner + col] =
                    make_double2(fc.to(v.y, 0), fc.to(v.x, 0));
            }
        };
        if (pl.nst == 0) {                                        // L = 1
            if (tid < C) store(0, c, z[c]);
        } else {
            fx_stages(z, pl, pl.nst - 1, lc, C, smem, shift);
            const int s = pl.nst - 1;
            fx_stage_any(z, pl, pl.s[s], lc, C, tid, nt, store,
                         [&](int) { return s && s == pl.shift_at ? fc.shift : 0; });
        }
        if (!REAL && FWD && valid && a.nc > 0)                    // the Nyquist entry
            for (int e = tid; e < C; e += nt)
                static_cast<double2*>(a.out)[(o * a.nc + a.nc / 2) * (long long)a.inner + col] = make_double2(0.0, 0.0);
    }
}

// ------------------------------------------------------------------------------------------------
// Chebyshev transforms of contiguous complex columns (Makhoul 1980: a DCT of length M by one FFT of
// length M), the conventions of cng_cheb_transform. A warp loads and stores a whole column (its scale
// needs no barrier); the stages run over all columns, rows padded by one element against conflicts.
template <bool FWD>
__device__ __forceinline__ void fx_cheb_body(unsigned bid, const FxChebArgs& a) {
    extern __shared__ __align__(16) unsigned char fx_sm[];
    __shared__ FxCol s_c[kFxCols];
    fx2* z = reinterpret_cast<fx2*>(fx_sm);
    const FxPlan& pl = a.plan;
    const int lc = a.lc, C = 1 << lc, CS = C > 1 ? C + 1 : 1, M = pl.L, N = a.N;
    const int tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
    const long long col0 = (long long)bid << lc;
    // item u of a column: the coefficients u and M - u (backward), or grid point u (forward)
    constexpr int NV = FWD ? 2 : 4;
    constexpr int H = FWD ? 8 : 4;
    const int items = FWD ? M : M / 2 + 1;
    const bool hold = items <= 32 * H;
    for (int t = tid >> 5; t < C; t += nw) {
        const bool valid = col0 + t < a.ncols;
        const double2* src = a.in + (col0 + t) * (FWD ? M : N);
        auto load = [&](int u, double* d) {
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = 0.0;
            if (!valid || u >= items) return;
            if (FWD || u < N) {
                const double2 v = src[u];
                d[0] = v.x;
                d[1] = v.y;
            }
            if constexpr (!FWD) {
                if (u > 0 && 2 * u < M && M - u < N) {
                    const double2 v = src[M - u];
                    d[2] = v.x;
                    d[3] = v.y;
                }
            }
        };
        double held[H][NV];
        int em = 0;
        unsigned T = 0;
        if (hold) {
#pragma unroll
            for (int u = 0; u < H; ++u) load(lane + 32 * u, held[u]);
#pragma unroll
            for (int u = 0; u < H; ++u)
#pragma unroll
                for (int q = 0; q < NV; ++q) em = max(em, fx_magnitude(held[u][q]));
        } else {
            for (int u = lane; u < items; u += 32) {
                load(u, held[0]);
#pragma unroll
                for (int q = 0; q < NV; ++q) em = max(em, fx_magnitude(held[0][q]));
            }
        }
        em = fx_column(__reduce_max_sync(0xffffffffu, em));
        FxCol fc;
        fc.bad = em == 0x7ff;
        if (hold) {
#pragma unroll
            for (int u = 0; u < H; ++u)
                if (lane + 32 * u < items)
#pragma unroll
                    for (int q = 0; q < NV; ++q) T += fx_weight(held[u][q], em);
        } else {
            for (int u = lane; u < items; u += 32) {
                load(u, held[0]);
#pragma unroll
                for (int q = 0; q < NV; ++q) T += fx_weight(held[0][q], em);
            }
        }
        T = __reduce_add_sync(0xffffffffu, T);
        {
            const FxScale f = fx_base(pl, em, T, 0);
            fc.base = f.base;
            fc.shift = f.shift;
        }
        if (lane == 0) s_c[t] = fc;
        auto convert = [&](int u, const double* d) {
            if (u >= items) return;
            fx f[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) f[q] = fc.bad ? 0 : fx_from(d[q], fc.base);
            if constexpr (FWD) {                                  // v_j = f_2j, v_{M-1-j} = f_{2j+1}
                z[(size_t)pl.in_pos[(u & 1) ? M - 1 - (u >> 1) : u >> 1] * CS + t] = fx2{f[0], f[1]};
            } else {
                // Z_k = (-1)^k / 2 e^{i pi k / 2M} (c_k - i c_{M-k}), Z_0 = c_0, as (y, x): inverse
                auto put = [&](int k, fx2 v) { z[(size_t)pl.in_pos[k] * CS + t] = fx2{v.y, v.x}; };
                const fx2 p = {f[0], f[1]}, q = {f[2], f[3]};
                if (u == 0) {
                    put(0, p);
                } else if (2 * u == M) {
                    put(u, fx_cmul(fx_sub_i(p, p), a.bq[u]));
                } else {
                    put(u, fx_cmul(fx_sub_i(p, q), a.bq[u]));
                    put(M - u, fx_cmul(fx_sub_i(q, p), a.bq[M - u]));
                }
            }
        };
        if (hold) {
#pragma unroll
            for (int u = 0; u < H; ++u) convert(lane + 32 * u, held[u]);
        } else {
            for (int u = lane; u < items; u += 32) {
                load(u, held[0]);
                convert(u, held[0]);
            }
        }
    }
    __syncthreads();
    fx_stages(z, pl, pl.nst, lc, CS, [&](int p, int c, fx2 v) { z[(size_t)p * CS + c] = v; },
              [&](int c) { return s_c[c].shift; });
    for (int t = tid >> 5; t < C; t += nw) {
        if (col0 + t >= a.ncols) break;
        const FxCol fc = s_c[t];
        double2* dst = a.out + (col0 + t) * (FWD ? N : M);
        if constexpr (FWD) {
            // c_k = s_k (Re (w_k (p + conj q)), Im (w_k (p - conj q))), p = Z_k, q = Z_{M-k}, the sign
            // and scale s_k in the table
            for (int k = lane; k < N; k += 32) {
                const fx2 p = z[(size_t)pl.out_pos[k] * CS + t], q = z[(size_t)pl.out_pos[k ? M - k : 0] * CS + t];
                const FxC wx = a.fq[2 * k], wy = a.fq[2 * k + 1], my = {-wy.h, -wy.l};
                const fx re = fx_mul2(p.x + q.x, wx, p.y - q.y, my);
                const fx im = fx_mul2(p.y + q.y, wx, p.x - q.x, wy);
                dst[k] = make_double2(fc.to(re, a.fshift), fc.to(im, a.fshift));
            }
        } else {
            // f_{2j} = z_j, f_{2j+1} = z_{M-1-j}
            for (int i = lane; i < M; i += 32) {
                const fx2 v = z[(size_t)pl.out_pos[(i & 1) ? M - 1 - (i >> 1) : i >> 1] * CS + t];
                dst[i] = make_double2(fc.to(v.y, 0), fc.to(v.x, 0));
            }
        }
    }
}

// 64 registers: these kernels wait on shared memory and on the products' latency, so resident warps count
// for more than a few spilled words. Channel 192 x 129 x 192 right-hand side by blocks of 256 threads an
// SM has registers for: 2 5.98 ms, 3 5.21, 4 5.03, 5 5.27; the ragged transforms 531, 483, 456, 471 us.
template <bool REAL, bool FWD>
__global__ void __launch_bounds__(kFxThreads, 4) k_fx_axis(const __grid_constant__ FxAxisArgs a) {
    fx_axis_body<REAL, FWD>(blockIdx.x, a);
}
template <bool REAL, bool FWD>
__global__ void __launch_bounds__(kFxThreads, 4) k_fx_axis_grp(const __grid_constant__ Grp<FxAxisArgs> g) {
    const int k = g.find(blockIdx.x);
    fx_axis_body<REAL, FWD>(blockIdx.x - g.start[k], g.a[k]);
}
template <bool FWD>
__global__ void __launch_bounds__(kFxThreads, 4) k_fx_cheb(const __grid_constant__ FxChebArgs a) {
    fx_cheb_body<FWD>(blockIdx.x, a);
}
template <bool FWD>
__global__ void __launch_bounds__(kFxThreads, 4) k_fx_cheb_grp(const __grid_constant__ Grp<FxChebArgs> g) {
    const int k = g.find(blockIdx.x);
    fx_cheb_body<FWD>(blockIdx.x - g.start[k], g.a[k]);
}

// ------------------------------------------------------------------------------------------------
// host: tables per device and length (a few hundred bytes to a few hundred KB, kept), launches

template <class T>
static const T* fx_upload(const std::vector<T>& h) {
    if (h.empty()) return nullptr;
    void* d = nullptr;
    CNG_CUDA(cudaMalloc(&d, sizeof(T) * h.size()));
    CNG_CUDA(cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
    return static_cast<const T*>(d);
}

struct FxDeviceTables {
    int device, L;
    FxPlan plan;
    const FxTw* bq = nullptr;                    // Chebyshev tables (even L)
    const FxC* fq = nullptr;
    int fshift = 0;
};

// c 2^shift in [1/2, 1)
static FxC fx_scale(long double c, int& shift) {
    shift = 0;
    while (c < 0.5L) {
        c *= 2;
        ++shift;
    }
    return fx_const(c);
}

static const FxDeviceTables& fx_device_tables(int L) {
    static std::mutex mu;
    static std::vector<std::unique_ptr<FxDeviceTables>> all;
    int dev = 0;
    CNG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    for (const auto& t : all)
        if (t->device == dev && t->L == L) return *t;
    int r = L;
    for (int p : {2, 3, 5})
        while (r > 0 && r % p == 0) r /= p;
    if (r != 1 || L < 1) throw InvalidArgument("FFT length " + std::to_string(L) + " must be 2^a 3^b 5^c");
    if (L > kFxMaxLen || fx_tables(L).plan.nst > kFxMaxStages)
        throw InvalidArgument("FFT length " + std::to_string(L) + " is too long for the shared-memory transforms");
    const FxTables T = fx_tables(L);
    auto d = std::make_unique<FxDeviceTables>();
    d->device = dev;
    d->L = L;
    d->plan = T.plan;
    d->plan.tw = fx_upload(T.tw);
    d->plan.in_pos = fx_upload(T.in_pos);
    d->plan.out_pos = fx_upload(T.out_pos);
    d->plan.k_of = fx_upload(T.k_of);
    if (L % 2 == 0) {
        const long double pi = 3.141592653589793238462643383279502884L;
        std::vector<FxTw> bq(L);
        std::vector<FxC> fq(2 * (size_t)L);
        long double s = 1.0L / L;
        while (s < 0.5L) {
            s *= 2;
            ++d->fshift;
        }
        for (int k = 0; k < L; ++k) {
            const long double x = cosl(pi * k / (2.0L * L)), y = sinl(pi * k / (2.0L * L));
            const long double h = (k & 1) ? -0.5L : 0.5L;
            bq[k] = fx_twiddle(h * x, h * y);
            const long double g = k == 0 ? 0.5L * s : ((k & 1) ? -s : s);     // (-1)^k / M, halved at k = 0
            fq[2 * (size_t)k] = fx_const(g * x);
            fq[2 * (size_t)k + 1] = fx_const(-g * y);
        }
        d->bq = fx_upload(bq);
        d->fq = fx_upload(fq);
    }
    all.push_back(std::move(d));
    return *all.back();
}

// Columns per block (1 << lc) and its shared memory. A block's columns are contiguous in memory: 8 of
// them make whole 128-byte lines (16 columns: fewer resident blocks, measured slower); fewer where a
// launch has too few columns to give every SM two blocks, or where the column is too long.
static int fx_log_cols(int L, long long cols, int maxseq, bool cheb) {
    int lc = 0;
    while (lc < 4 && (2 << lc) <= (maxseq > 0 ? maxseq : 8)) ++lc;
    if (maxseq <= 0)
        while (lc > 0 && (cols >> lc) < 2LL * sm_count()) --lc;
    while (lc > 0 && (size_t)L * ((1 << lc) + (cheb ? 1 : 0)) * sizeof(fx2) > kFxSmem) --lc;
    if ((size_t)L * sizeof(fx2) > kFxSmem) throw InvalidArgument("FFT length too long for the shared-memory transforms");
    return lc;
}
// threads of a block: about one radix-8 butterfly each
static int fx_threads(int L, int lc, int threads) {
    if (threads <= 0) threads = ((((L << lc) + 7) / 8 + 31) / 32) * 32;
    return std::min(std::max(threads, 64), kFxThreads);
}

template <class A, class K1, class KG>
static void fx_launch(const std::vector<A>& args, const std::vector<unsigned>& blocks, K1 one, KG grp, int threads,
                      size_t smem, cudaStream_t st) {
    ensure_smem_attr((const void*)one, (int)kFxSmem);
    if (args.size() == 1) {
        if (blocks[0]) one<<<blocks[0], threads, smem, st>>>(args[0]);
        CNG_LAUNCH("fixed-point transform");
        return;
    }
    ensure_smem_attr((const void*)grp, (int)kFxSmem);
    launch_groups(args, blocks, [&](const Grp<A>& g, unsigned total) {
        grp<<<total, threads, smem, st>>>(g);
        CNG_LAUNCH("fixed-point transform (group)");
    });
}

static unsigned fx_blocks(long long n) {
    if (n > 0x7fffffffLL) throw InvalidArgument("transform batch too large for one launch");
    return (unsigned)n;
}

void fx_cheb(const std::vector<FxChebJob>& jobs, bool forward, cudaStream_t st, int threads) {
    std::vector<FxChebArgs> args;
    std::vector<unsigned> blocks;
    size_t smem = 0;
    int nt = 0;
    for (const auto& j : jobs) {
        if (j.M % 2) throw InvalidArgument("Chebyshev grid size must be even");
        const FxDeviceTables& t = fx_device_tables(j.M);
        const int lc = fx_log_cols(j.M, j.ncols, j.maxseq, true);
        args.push_back(FxChebArgs{j.in, j.out, j.ncols, j.N, lc, t.plan, t.bq, t.fq, t.fshift});
        blocks.push_back(fx_blocks((j.ncols + (1 << lc) - 1) >> lc));
        smem = std::max(smem, (size_t)j.M * ((1 << lc) + (lc ? 1 : 0)) * sizeof(fx2));
        nt = std::max(nt, fx_threads(j.M, lc, threads));
    }
    if (forward) fx_launch(args, blocks, k_fx_cheb<true>, k_fx_cheb_grp<true>, nt, smem, st);
    else fx_launch(args, blocks, k_fx_cheb<false>, k_fx_cheb_grp<false>, nt, smem, st);
}

void fx_axis(const std::vector<FxAxisJob>& jobs, bool real, bool forward, cudaStream_t st, int threads) {
    std::vector<FxAxisArgs> args;
    std::vector<unsigned> blocks;
    size_t smem = 0;
    int nt = 0;
    for (const auto& j : jobs) {
        const FxDeviceTables& t = fx_device_tables(j.L);
        const long long cols = real ? (j.inner + 1) / 2 : j.inner;
        const int lc = fx_log_cols(j.L, cols * j.outer, j.maxseq, false);
        // a caller's reals may start 8 bytes off (a slice of a buffer)
        const int wide = j.inner % 2 == 0 && reinterpret_cast<uintptr_t>(j.out) % 16 == 0;
        FxAxisArgs a{j.in, j.out, j.outer, j.inner, std::max(j.ncompact, 0), lc, t.plan, FxC{}, 0, wide, j.ex};
        a.scale = fx_scale(1.0L / ((real ? 2.0L : 1.0L) * j.L), a.shift);
        args.push_back(a);
        blocks.push_back(fx_blocks(j.outer * ((cols + (1 << lc) - 1) >> lc)));
        smem = std::max(smem, ((size_t)j.L << lc) * sizeof(fx2));
        nt = std::max(nt, fx_threads(j.L, lc, threads));
    }
    if (real && forward) fx_launch(args, blocks, k_fx_axis<true, true>, k_fx_axis_grp<true, true>, nt, smem, st);
    else if (real) fx_launch(args, blocks, k_fx_axis<true, false>, k_fx_axis_grp<true, false>, nt, smem, st);
    else if (forward) fx_launch(args, blocks, k_fx_axis<false, true>, k_fx_axis_grp<false, true>, nt, smem, st);
    else fx_launch(args, blocks, k_fx_axis<false, false>, k_fx_axis_grp<false, false>, nt, smem, st);
}

}  // namespace cng
