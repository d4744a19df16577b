// Phases of complex systems that are real up to powers of i (real_form.cuh).
#include "real_form.cuh"

#include <algorithm>

namespace cng {

// bit 0: a nonzero real part at this slot in some sampled system, bit 1: a nonzero imaginary part
__global__ void k_entry_class(const zd* __restrict__ a, long long slots, int batch, int stride,
                              unsigned char* __restrict__ out) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < slots;
         q += (long long)gridDim.x * blockDim.x) {
        unsigned char c = 0;
        for (int k = 0; k < batch && c != 3; k += stride) {
            const zd v = a[(size_t)k * slots + q];
            c |= (v.re != 0.0 ? 1 : 0) | (v.im != 0.0 ? 2 : 0);
        }
        out[q] = c;
    }
}

bool find_phases(const zd* ab, const zd* vt, int batch, int n, int r, int kv, int ldab, cudaStream_t st,
                 std::vector<unsigned char>& row, std::vector<unsigned char>& col) {
    const long long na = (long long)n * ldab, nv = (long long)r * n;
    std::vector<unsigned char> cls((size_t)(na + nv));
    unsigned char* d = static_cast<unsigned char*>(dev_alloc(cls.size()));
    try {
        const int stride = std::max(1, batch / 256);
        k_entry_class<<<ceil_div(na, 128), 128, 0, st>>>(ab, na, batch, stride, d);
        CNG_LAUNCH("k_entry_class");
        if (nv) {
            k_entry_class<<<ceil_div(nv, 128), 128, 0, st>>>(vt, nv, batch, stride, d + na);
            CNG_LAUNCH("k_entry_class");
        }
        CNG_CUDA(cudaMemcpyAsync(cls.data(), d, cls.size(), cudaMemcpyDeviceToHost, st));
        CNG_CUDA(cudaStreamSynchronize(st));
    } catch (...) {
        dev_free(d);
        throw;
    }
    dev_free(d);
    // Phases of rows (nodes 0 .. n-1) and columns (n ..): an entry joins equal (real) or different (imaginary)
    // ones. Sets of joined nodes, each with its phase against the set's root.
    std::vector<int> up((size_t)2 * n);
    std::vector<unsigned char> phase((size_t)2 * n, 0);          // against `up`
    for (int u = 0; u < 2 * n; ++u) up[u] = u;
    auto root = [&](int u) {
        unsigned char p = 0;
        int v = u;
        for (; up[v] != v; v = up[v]) p ^= phase[v];
        while (up[u] != v) {                                     // the path shortened
            const int w = up[u];
            const unsigned char q = phase[u];
            up[u] = v;
            phase[u] = p;
            p ^= q;
            u = w;
        }
        return v;
    };
    auto join = [&](int i, int j, unsigned char c) {
        const int u = root(i), v = root(n + j);                  // i and n + j now hang on their roots
        const unsigned char want = (unsigned char)((c >> 1) ^ phase[i] ^ phase[n + j]);
        if (u == v) return want == 0;
        up[u] = v;
        phase[u] = want;
        return true;
    };
    for (int j = 0; j < n; ++j)
        for (int q = 0; q < ldab; ++q) {
            const unsigned char c = cls[(size_t)j * ldab + q];
            const int i = j + q - kv;
            if (c == 3 || (c && i >= 0 && i < n && !join(i, j, c))) return false;
        }
    for (int a = 0; a < r; ++a)
        for (int j = 0; j < n; ++j) {
            const unsigned char c = cls[(size_t)na + (size_t)a * n + j];
            if (c == 3 || (c && !join(a, j, c))) return false;
        }
    for (int u = 0; u < 2 * n; ++u) root(u);
    for (int u = 0; u < 2 * n; ++u)
        if (up[u] == u) phase[u] = 0;
    row.assign(phase.begin(), phase.begin() + n);
    col.assign(phase.begin() + n, phase.end());
    return true;
}

}  // namespace cng
