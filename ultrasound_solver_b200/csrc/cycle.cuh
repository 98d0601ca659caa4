// One restart cycle's Arnoldi steps in a single launch (cycle.cu).
#pragma once

#include "cycle_split.h"
#include "krylov.cuh"

namespace usv {

// Launch geometry of the cycle kernel for right-hand sides of sizes[b] nodes;
// ctas = 0: this solve keeps one launch per Arnoldi pass.
struct CyclePlan {
    const void* fn = nullptr;
    int ctas = 0;
    size_t smem = 0;
};
template <typename R, typename S, bool MS>
cudaError_t cycle_plan(int m, const long long* sizes, int nrhs, int sms, CyclePlan& plan);

}  // namespace usv
