// The scheduled solve (flow_solve.cu): built from a factorization, launched for several buckets at once.
#pragma once

#include <memory>
#include <vector>

#include "common.cuh"
#include "solve_io.cuh"

namespace cng {

// The most bytes of operations of a system per column; more are refused (memory.py plans them). A slot takes
// 384 bytes with one right-hand side per factor, 192 with two, 96 with four (all its operations, used or
// not), so this is a limit on slots: 1.04 a column for real systems, 2.08 for complex ones, 4.2 for shared pairs.
// It is set by memory: what the planner counts for the steps' systems stays below the compact streams (about 790
// bytes a column on the channel), and they fit it (slots a column: singles 0.9, Burgers 1.2, RB 1.35, the
// channel's pairs 1.9). It is not where the time crosses: a real band that couples both parities takes 2 slots
// a column and is refused from n of about 70 on, though its operations (700 bytes a column, its band 24) would
// solve 31 systems of n = 200 in 26 us where the band kernel takes 69, and 2048 in 69 where it takes 123.
constexpr int kFlowColumnBytes = 400;

struct FlowSource {                      // the factored handle's arrays (banded.cu)
    int dtype, batch, n, r, kl, ku, ldab;
    const void* ab;
    const int* ipiv;
    const void* vt;
    const void* w;
    const void* slu;
    const int* spiv;
    const int* perm;
    bool in_order;                       // perm is the identity
    const unsigned char* rowp;           // phases of the real form (complex handles)
    const unsigned char* colp;
    const unsigned char* flip_r;         // a shared pair's signs (NULL: no partner)
    const unsigned char* flip_c;
    bool fp32;                           // also the FP32 copies (mixed form)
    int lanes;                           // lanes of a border sum: 16 or 32
    size_t most;                         // most bytes of operations (0: what the device has)
};

struct FlowForm {
    int n = 0, batch = 0, dtype = 0, lanes = 0;
    int rows = 0;                        // rows of a system's vector: n, the border's sums, a zero
    int ncr = 0;                         // right-hand sides of a factor: components x (system, partner)
    int chunks = 0;                      // largest number of chunks of operations of a system
    size_t sb[2] = {0, 0};               // bytes of a system: FP64, FP32
    size_t used[2] = {0, 0};             // bytes that a solve of every system reads of them
    unsigned char* data[2] = {nullptr, nullptr};
    int* nchunk = nullptr;               // per system
    unsigned short* row = nullptr;       // [batch][n]: the name of each row
    const int* perm = nullptr;           // NULL: the rows as they come
    unsigned char* flags = nullptr;      // [2][n]: rows' and columns' phase | partner's sign << 1
    ~FlowForm();
    FlowForm() = default;
    FlowForm(const FlowForm&) = delete;
    FlowForm& operator=(const FlowForm&) = delete;
};

// Throws InvalidArgument where the form does not apply (size, fill, or values that are not real up to
// the phases) or takes more than `most` bytes. The handles' builds run side by side after `st`'s work, and
// are waited for.
std::vector<std::unique_ptr<FlowForm>> flow_build(const std::vector<FlowSource>& sources, cudaStream_t st);

struct FlowJob {
    const FlowForm* form;
    SolveIo io, io2;                     // io2: the partner (rhs NULL: none)
    int s0, s1;                          // systems solved
};
void flow_solve(const std::vector<FlowJob>& jobs, int io_kind, cudaStream_t st);

}  // namespace cng
