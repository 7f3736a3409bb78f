// The reference's kernel launchers (core/src/gpu/cuda_pdhg.cu:155-203) with
// their exact argument lists: separate int32 index and float value arrays,
// device pointers, a caller stream.  The reference's host driver binds them at
// core/src/gpu/gpu_solver.cpp:18-40.  Updates are the reference's element
// formulas with unfused float operations.
#include <algorithm>

#include "common.cuh"
#include "compat.cuh"
#include "spmv.cuh"

namespace sihg {

__device__ __forceinline__ float split_dot(const int* __restrict__ idx, const float* __restrict__ val, int beg,
                                           int end, int lane0, int L, const float* __restrict__ vec) {
    float s0 = 0.f, s1 = 0.f;
    unsigned k = (unsigned)beg + lane0;  // (unsigned: a step may end past 2^31 - 1)
    const unsigned last = end;
    for (; (int)(last - k) > L; k += 2 * L) {
        s0 = fmaf(__ldg(val + k), __ldg(vec + __ldg(idx + k)), s0);
        s1 = fmaf(__ldg(val + k + L), __ldg(vec + __ldg(idx + k + L)), s1);
    }
    if ((int)(last - k) > 0) s0 = fmaf(__ldg(val + k), __ldg(vec + __ldg(idx + k)), s0);
    return s0 + s1;
}

// Segments summed in place by groups of L lanes (few or long segments), by the
// first `blocks` blocks.
__device__ __forceinline__ void spmv_by_groups(int nseg, const int* __restrict__ ptr, const int* __restrict__ idx,
                                               const float* __restrict__ val, const float* __restrict__ vec,
                                               float* __restrict__ out, int L, int blocks) {
    if (blockIdx.x >= blocks) return;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), gpw = 32 / L;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (blocks * blockDim.x) >> 5;
    for (unsigned base = wid * gpw; base < (unsigned)nseg; base += nw * gpw) {  // unsigned: nseg + a turn may pass 2^31
        const unsigned r = base + lane / L;
        float s = 0.f;
        if (r < (unsigned)nseg) s = split_dot(idx, val, ptr[r], ptr[r + 1], sub, L, vec);
        for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_down_sync(FULL_MASK, s, o, L);
        if (r < (unsigned)nseg && sub == 0) out[r] = s;
    }
}

__device__ __forceinline__ int ld_stream(const int* p) {
    int v;
    asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// s + c <- s + c + v, c the compensation
__device__ __forceinline__ void comp_add(float& s, float& c, float v) {
    float t, e;
    two_sum(s, v, t, e);
    s = t;
    c = __fadd_rn(c, e);
}

// Many short segments: a warp takes 32 consecutive segments and reads their
// entries as one stream, eight per lane in flight, whatever the segments'
// lengths (products go to shared memory; Greathouse and Daga's CSR-stream,
// SC14); then each lane sums its own segment, and the warp together the ones
// longer than kLong.  Groups of lanes leave the lanes of short segments idle
// while the group of a long one works.  What bounds it is the gathers: one
// cache line each, which the L1 takes one at a time per SM (12M of them: 46 us).
//
// The products are rounded on their way through shared memory, so the sums are
// compensated: relative error 3.5e-8 at any length, against 3.9e-8 (3 entries) to
// 6.2e-8 (31) of fused multiply-adds by groups of lanes and 4.2e-8 to 8.1e-8 of
// plain sums of the products.  Values and gathered entries side by side in shared
// memory, for fused multiply-adds here too, leave the gathers too little L1.
//
// 1M segments of 12 entries (12M) and 500k of 24, us by groups / plain sums / so: equal
// lengths 53 / 48 / 48 and 54 / 49 / 49, lengths by a power law (2 to 2000) 147 / 58 / 62
// and 130 / 66 / 72.  64 warps per SM (32 registers; the pointers are read again
// after the gathers to stay within them) matter most: 48 warps 5 to 12 % more;
// windows of 256 / 640 products 20 / 10 %, 16 entries a lane in flight 32 %; kLong 24 / 32:
// 28 / 7 % more on rows of 24.
constexpr int kLong = 48;
__device__ __forceinline__ void spmv_by_stream(int nseg, const int* __restrict__ ptr, const int* __restrict__ idx,
                                               const float* __restrict__ val, const float* __restrict__ vec,
                                               float* __restrict__ out, float* prod) {
    constexpr int kU = 8;
    const int lane = threadIdx.x & 31;
    // to every block's first warp first, so that the blocks have even shares
    const int wid = blockIdx.x + gridDim.x * (threadIdx.x >> 5), nw = (gridDim.x * blockDim.x) >> 5;
    const unsigned last = nseg;
    for (unsigned base = wid * 32u; base < last; base += nw * 32u) {
        const unsigned end = ptr[min(base + 32u, last)];
        float s = 0.f, c = 0.f;
        // (unsigned: the last window of 2^31 - 1 entries ends past them)
        for (unsigned w = ptr[base]; (int)(end - w) > 0; w += kWindow) {
            const int n = min(kWindow, (int)(end - w));
            for (int k0 = lane; k0 < n; k0 += 32 * kU) {
                int i[kU];
                float a[kU], g[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const bool on = k0 + 32 * u < n;
                    i[u] = on ? ld_stream(idx + w + k0 + 32 * u) : -1;
                    a[u] = on ? ld_stream(val + w + k0 + 32 * u) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) g[u] = i[u] >= 0 ? __ldg(vec + i[u]) : 0.f;
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (i[u] >= 0) prod[k0 + 32 * u] = a[u] * g[u];
            }
            __syncwarp();
            // this lane's segment and its part of the window
            const unsigned r = base + lane;
            const int b = ptr[min(r, last)] - (int)w, e = ptr[min(r + 1, last)] - (int)w;
            const int lo = max(b, 0), hi = min(e, n);
            if (e - b <= kLong)
                for (int k = lo; k < hi; ++k) comp_add(s, c, prod[k]);
            for (unsigned m = __ballot_sync(FULL_MASK, e - b > kLong); m; m &= m - 1) {
                const int from = __ffs(m) - 1;
                const int lo1 = __shfl_sync(FULL_MASK, lo, from), hi1 = __shfl_sync(FULL_MASK, hi, from);
                float p = 0.f, pc = 0.f;
                for (int k = lo1 + lane; k < hi1; k += 32) comp_add(p, pc, prod[k]);
                __syncwarp();
                group_sum2(p, pc, 32);
                p = __shfl_sync(FULL_MASK, p, 0);
                pc = __shfl_sync(FULL_MASK, pc, 0);
                if (lane == from) {
                    comp_add(s, c, p);
                    c += pc;
                }
            }
            __syncwarp();
        }
        // (an infinite sum has no compensation)
        if (base + lane < last) out[base + lane] = isfinite(s) ? s + c : s;
    }
}

// Lanes per segment from the mean segment length, from the last pointer: read
// on the device, so that no launch has to ask the host for it.  By stream from
// kStreamSegs segments on, where every SM has several warps of 32, and below a
// mean of 32 (L < 16), where equal lengths are no slower by it at any count.  us by
// groups / by stream for segments of 20, 28, 36 and 56 entries, back to back: 60,000
// equal ones 8.7 / 8.9, 11.3 / 11.1, 11.9 / 13.9, 17 / 48; 400,000 equal ones 38 / 36,
// 56 / 47, 74 / 59, 104 / 186 (past kLong the warp sums each alone); by a power law 60,000
// 35 / 22, 48 / 30, 40 / 42, 58 / 76 and 400,000 80 / 48, 124 / 68, 148 / 90, 224 / 154.
__global__ void __launch_bounds__(kSplitThreads, 8) split_spmv_kernel(int nseg, const int* __restrict__ ptr,
                                                                      const int* __restrict__ idx,
                                                                      const float* __restrict__ val,
                                                                      const float* __restrict__ vec,
                                                                      float* __restrict__ out, int group_blocks) {
    extern __shared__ float prod[];  // [warps that have segments by stream][kWindow]
    chain_wait_for(ptr, idx, val, vec, out);
    const long long nnz = ptr[nseg];
    int L = 1;
    while (L < 32 && 4ll * L * nseg <= nnz) L *= 2;
    if (nseg >= kStreamSegs && L < 16)
        spmv_by_stream(nseg, ptr, idx, val, vec, out, prod + kWindow * (threadIdx.x >> 5));
    else
        spmv_by_groups(nseg, ptr, idx, val, vec, out, L, group_blocks);
}

__global__ void compat_primal_kernel(int n, const float* __restrict__ tau, const float* __restrict__ c,
                                     const float* __restrict__ aty, const float* __restrict__ l,
                                     const float* __restrict__ u, float* __restrict__ x,
                                     float* __restrict__ xbar) {
    chain_wait_for(tau, c, aty, l, u, x, xbar);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const float x_old = x[j];
        float x_new = __fsub_rn(x_old, __fmul_rn(tau[j], __fadd_rn(c[j], aty[j])));
        if (x_new < l[j]) x_new = l[j];
        if (x_new > u[j]) x_new = u[j];
        x[j] = x_new;
        xbar[j] = __fsub_rn(__fmul_rn(2.0f, x_new), x_old);
    }
}

__global__ void compat_dual_kernel(int m, const float* __restrict__ sigma, const float* __restrict__ axbar,
                                   const float* __restrict__ rl, const float* __restrict__ ru,
                                   float* __restrict__ y) {
    chain_wait_for(sigma, axbar, rl, ru, y);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const float sig = sigma[i];
        const float w = __fadd_rn(axbar[i], y[i] / sig);
        float p = w;
        if (p < rl[i]) p = rl[i];
        if (p > ru[i]) p = ru[i];
        y[i] = __fmul_rn(sig, __fsub_rn(w, p));
    }
}

__global__ void compat_copy_kernel(int n, const float* __restrict__ x, float* __restrict__ xbar) {
    chain_wait_for(x, xbar);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) xbar[j] = x[j];
}

__global__ void compat_residuals_kernel(int m, int n, const float* __restrict__ ax, const float* __restrict__ rl,
                                        const float* __restrict__ ru, float* __restrict__ row_out,
                                        const float* __restrict__ x, const float* __restrict__ c,
                                        const float* __restrict__ aty, const float* __restrict__ l,
                                        const float* __restrict__ u, const float* __restrict__ tau,
                                        float* __restrict__ col_out) {
    chain_wait_for(ax, rl, ru, row_out, x, c, aty, l, u, tau, col_out);
    const int stride = gridDim.x * blockDim.x;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
        const float xj = x[j], step = tau[j];
        float proj = __fsub_rn(xj, __fmul_rn(step, __fadd_rn(c[j], aty[j])));
        if (proj < l[j]) proj = l[j];
        if (proj > u[j]) proj = u[j];
        col_out[j] = fabsf(__fsub_rn(xj, proj)) / fmaxf(1e-4f, step);
    }
    // rows from the other end of the grid, whose blocks have fewer columns
    for (int i = (gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += stride) {
        const float a = ax[i];
        float viol = 0.0f;
        if (rl[i] > -1e15f && a < rl[i]) viol = fmaxf(viol, __fsub_rn(rl[i], a));
        if (ru[i] < 1e15f && a > ru[i]) viol = fmaxf(viol, __fsub_rn(a, ru[i]));
        row_out[i] = viol;
    }
}

static int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

static int grid_for(int n) { return std::max(1, std::min((n + 255) / 256, sm_count() * 8)); }

static int split_spmv(int nseg, const int* ptr, const int* idx, const float* val, const float* vec, float* out,
                      void* stream) {
    if (nseg < 0) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "negative dimension");
    if (nseg == 0) return SIH_PDHG_OK;
    if (!ptr || !out || !vec) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "NULL device pointer");
    const SplitLaunch g = split_launch(nseg, sm_count());
    SIHG_CUDA(launch_chained(split_spmv_kernel, g.blocks, g.threads, g.smem, static_cast<cudaStream_t>(stream), nseg, ptr,
                             idx, val, vec, out, g.group_blocks));
    return SIH_PDHG_OK;
}

}  // namespace sihg

using namespace sihg;

// Every launcher runs inside guarded(): the error messages can throw, and no
// exception may cross the C ABI.  The kernels are chained (launch_chained): a
// launcher's kernel is scheduled while the one before it in the stream ends, and
// waits for it on the device.
extern "C" int sih_pdhg_launch_csr_spmv(int m, const int* d_row_ptr, const int* d_col_ind, const float* d_values,
                                        const float* d_x, float* d_y, void* stream) {
    return guarded([&] { return split_spmv(m, d_row_ptr, d_col_ind, d_values, d_x, d_y, stream); });
}

extern "C" int sih_pdhg_launch_csc_spmv(int n, const int* d_col_ptr, const int* d_row_ind, const float* d_values,
                                        const float* d_y, float* d_z, void* stream) {
    return guarded([&] { return split_spmv(n, d_col_ptr, d_row_ind, d_values, d_y, d_z, stream); });
}

extern "C" int sih_pdhg_launch_primal_update(int n, const float* d_tau, const float* d_c, const float* d_AT_y,
                                             const float* d_l, const float* d_u, float* d_x, float* d_x_bar,
                                             void* stream) {
    return guarded([&]() -> int {
        if (n < 0) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "negative dimension");
        if (n == 0) return SIH_PDHG_OK;
        SIHG_CUDA(launch_chained(compat_primal_kernel, grid_for(n), 256, 0, (cudaStream_t)stream, n, d_tau, d_c, d_AT_y,
                                 d_l, d_u, d_x, d_x_bar));
        return SIH_PDHG_OK;
    });
}

extern "C" int sih_pdhg_launch_dual_update(int m, const float* d_sigma, const float* d_A_xbar, const float* d_row_l,
                                           const float* d_row_u, float* d_y, void* stream) {
    return guarded([&]() -> int {
        if (m < 0) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "negative dimension");
        if (m == 0) return SIH_PDHG_OK;
        SIHG_CUDA(launch_chained(compat_dual_kernel, grid_for(m), 256, 0, (cudaStream_t)stream, m, d_sigma, d_A_xbar,
                                 d_row_l, d_row_u, d_y));
        return SIH_PDHG_OK;
    });
}

extern "C" int sih_pdhg_launch_restart(int n, const float* d_x, float* d_x_bar, void* stream) {
    return guarded([&]() -> int {
        if (n < 0) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "negative dimension");
        if (n == 0) return SIH_PDHG_OK;
        SIHG_CUDA(launch_chained(compat_copy_kernel, grid_for(n), 256, 0, (cudaStream_t)stream, n, d_x, d_x_bar));
        return SIH_PDHG_OK;
    });
}

extern "C" int sih_pdhg_launch_residuals(int m, int n, const float* d_Ax, const float* d_row_l, const float* d_row_u,
                                         float* d_row_viols, const float* d_x, const float* d_c, const float* d_AT_y,
                                         const float* d_l, const float* d_u, const float* d_tau, float* d_col_viols,
                                         void* stream) {
    return guarded([&]() -> int {
        if (m < 0 || n < 0) return fail(SIH_PDHG_ERR_INVALID_ARGUMENT, "negative dimension");
        if (m == 0 && n == 0) return SIH_PDHG_OK;
        SIHG_CUDA(launch_chained(compat_residuals_kernel, grid_for(std::max(m, n)), 256, 0, (cudaStream_t)stream, m, n,
                                 d_Ax, d_row_l, d_row_u, d_row_viols, d_x, d_c, d_AT_y, d_l, d_u, d_tau, d_col_viols));
        return SIH_PDHG_OK;
    });
}
