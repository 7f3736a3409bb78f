// Kernels of the reference-compatible launchers (compat.cu), declared for
// reuse by other translation units.
#pragma once

#include <algorithm>

namespace sihg {

// out[s] = sum of val[k] vec[idx[k]] over the entries of segment s.
__global__ void split_spmv_kernel(int nseg, const int* __restrict__ ptr, const int* __restrict__ idx,
                                  const float* __restrict__ val, const float* __restrict__ vec,
                                  float* __restrict__ out);
constexpr int kSplitThreads = 128;
// From this many segments on split_spmv_kernel may take 32 segments a warp.
constexpr int kStreamSegs = 1 << 15;
// Blocks of split_spmv_kernel.  Many segments: a warp per 32 of them, as many
// blocks as that takes, so that the hardware hands out new blocks as old ones
// end (columns of Zipf lengths).  Few: a warp per segment, what 32 lanes a segment would
// need (the kernel takes fewer where the mean length says so), at most 16 a SM.
inline int split_grid(int nseg, int sms) {
    constexpr int kWarps = kSplitThreads / 32;
    if (nseg >= kStreamSegs) return (nseg + 32 * kWarps - 1) / (32 * kWarps);
    return std::max(1, std::min((nseg + kWarps - 1) / kWarps, sms * 16));
}

// Column measures (blocks first) and row violations of a point, one launch.
__global__ void compat_residuals_kernel(int m, int n, const float* __restrict__ ax, const float* __restrict__ rl,
                                        const float* __restrict__ ru, float* __restrict__ row_out,
                                        const float* __restrict__ x, const float* __restrict__ c,
                                        const float* __restrict__ aty, const float* __restrict__ l,
                                        const float* __restrict__ u, const float* __restrict__ tau,
                                        float* __restrict__ col_out);

}  // namespace sihg
