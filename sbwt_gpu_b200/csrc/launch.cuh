// launch.cuh -- launch of a search kernel on a stream.
#pragma once
#include "internal.h"

namespace sbwt {

// Launches a search kernel with the L2 access-policy window of the index's
// rank lines, where one applies (l2_window).
template <class K, class R>
int launch_kernel(K kern, u32 blocks, u32 threads, cudaStream_t s, const sbwt_index *ix, const R &rk,
                  const SearchArgs &a) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.numAttrs = 0;
    if (l2_window(ix, a.walk, &attr[0].val.accessPolicyWindow)) {
        attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    SBWT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, rk, a));
    return 0;
}

}  // namespace sbwt
