// The FP64 transforms (fixed_transforms.cu): launchers for single problems and for groups of problems
// of different sizes (one launch per kMaxGrp of them). `maxseq` and `threads` as cng_rhs_set_tuning
// (0: the defaults); neither changes a result.
#pragma once

#include <vector>

#include "common.cuh"
#include "expand.cuh"

namespace cng {

struct FxChebJob {
    const double2* in;
    double2* out;
    long long ncols;
    int N, M, maxseq;
};
struct FxAxisJob {
    const void* in;
    void* out;
    long long outer;
    int inner, ncompact, L, maxseq;        // ncompact: Nc (complex transform) or K (real transform)
    Expand<double> ex;
};

void fx_cheb(const std::vector<FxChebJob>& jobs, bool forward, cudaStream_t st, int threads);
void fx_axis(const std::vector<FxAxisJob>& jobs, bool real, bool forward, cudaStream_t st, int threads);

}  // namespace cng
