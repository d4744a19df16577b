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
    // two-colour rows (nodes 0 .. n-1) and columns (n ..): an entry joins equal (real) or different
    // (imaginary) phases
    std::vector<std::vector<std::pair<int, unsigned char>>> adj((size_t)2 * n);
    auto edge = [&](int i, int j, unsigned char c) {
        adj[i].push_back({n + j, (unsigned char)(c >> 1)});
        adj[n + j].push_back({i, (unsigned char)(c >> 1)});
    };
    for (int j = 0; j < n; ++j)
        for (int q = 0; q < ldab; ++q) {
            const unsigned char c = cls[(size_t)j * ldab + q];
            const int i = j + q - kv;
            if (c == 3) return false;
            if (c && i >= 0 && i < n) edge(i, j, c);
        }
    for (int a = 0; a < r; ++a)
        for (int j = 0; j < n; ++j) {
            const unsigned char c = cls[(size_t)na + (size_t)a * n + j];
            if (c == 3) return false;
            if (c) edge(a, j, c);
        }
    std::vector<signed char> phase((size_t)2 * n, -1);
    std::vector<int> stack;
    for (int s = 0; s < 2 * n; ++s) {
        if (phase[s] >= 0) continue;
        phase[s] = 0;
        stack.assign(1, s);
        while (!stack.empty()) {
            const int u = stack.back();
            stack.pop_back();
            for (const auto& e : adj[u]) {
                const signed char want = (signed char)(phase[u] ^ e.second);
                if (phase[e.first] < 0) {
                    phase[e.first] = want;
                    stack.push_back(e.first);
                } else if (phase[e.first] != want) {
                    return false;
                }
            }
        }
    }
    row.assign(phase.begin(), phase.begin() + n);
    col.assign(phase.begin() + n, phase.end());
    return true;
}

}  // namespace cng
