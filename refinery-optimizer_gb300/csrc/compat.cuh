// Kernels of the reference-compatible launchers (compat.cu), declared for
// reuse by other translation units.
#pragma once

#include <algorithm>

namespace sihg {

// out[s] = sum of val[k] vec[idx[k]] over the entries of segment s.
__global__ void split_spmv_kernel(int nseg, const int* __restrict__ ptr, const int* __restrict__ idx,
                                  const float* __restrict__ val, const float* __restrict__ vec,
                                  float* __restrict__ out, int group_blocks);
constexpr int kSplitThreads = 256;  // most of a block
// From this many segments on split_spmv_kernel may take 32 segments a warp.
constexpr int kStreamSegs = 1 << 15;
constexpr int kWindow = 512;  // products of a warp at a time, there
// Launch of split_spmv_kernel, which learns on the device whether it goes by
// groups of lanes or by stream.  By groups it wants a warp per segment, what 32
// lanes a segment would need (it takes fewer where the mean length says so), as
// far as the SMs hold them, 64 warps each, and no more: further blocks would make
// a second wave (400,000 equal segments of 33 / 70 entries 88 / 169 us with it, 70 / 140
// without; by a power law 122 / 196 and 134 / 181).  By stream a warp per 32
// segments: with more of those than the SMs hold, blocks of four warps, which the
// hardware hands out as others end (columns of Zipf lengths); below, what the groups
// want, in blocks of eight, of which the stream leaves some warps idle: only the
// others have a window, because its shared memory is missing in the groups' L1.
// 40,000 / 100,000 / 250,000 segments of 70 entries (groups) with a warp per 32 segments
// everywhere 38.2 / 48.1 / 105, with a window for every warp 14.8 / 33.0 / 86.5, so 13.8 /
// 32.3 / 85.0 us; of 24 (stream) 8.7 / 14.8 / 31.9, 8.1 / 14.7 / 28.1 and 7.9 / 13.8 / 27.6.
struct SplitLaunch {
    int blocks, threads, smem;
    int group_blocks;  // that the groups use
};
inline SplitLaunch split_launch(int nseg, int sms) {
    const int units = (nseg - 1) / 32 + 1;
    const bool many = nseg >= kStreamSegs && units > 64 * sms;
    const int warps = many ? 4 : kSplitThreads / 32;
    const int held = std::max(1, 64 * sms / warps);
    const int blocks = many ? (units - 1) / warps + 1 : std::min((nseg - 1) / warps + 1, held);
    const int windows = nseg >= kStreamSegs ? (units - 1) / blocks + 1 : 0;
    return SplitLaunch{blocks, 32 * warps, (int)sizeof(float) * kWindow * windows, std::min(blocks, held)};
}

// Column measures (blocks first) and row violations of a point, one launch.
__global__ void compat_residuals_kernel(int m, int n, const float* __restrict__ ax, const float* __restrict__ rl,
                                        const float* __restrict__ ru, float* __restrict__ row_out,
                                        const float* __restrict__ x, const float* __restrict__ c,
                                        const float* __restrict__ aty, const float* __restrict__ l,
                                        const float* __restrict__ u, const float* __restrict__ tau,
                                        float* __restrict__ col_out);

}  // namespace sihg
