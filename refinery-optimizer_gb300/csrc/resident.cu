// Resident step form: the steps between two evaluations of an LP whose matrix,
// vectors and controller state all fit in the shared memory of one thread-block
// cluster (one block for the smallest), a cluster per instance of a batch.
//
// Small LPs are bound by latency: in the other forms every step crosses the
// whole chip two or three times (kernel boundaries or grid barriers, 1.5 us
// each) and every gather goes to L2.  Here a step touches no global memory:
// the block's share of both sides of the matrix stays in shared memory for the
// whole launch, every block of the cluster holds a copy of x' and y' that it
// gathers from, owners push their new entries to all copies through
// distributed shared memory, and the phases are separated by the hardware
// cluster barrier.  (Gathering from another block's shared memory instead was
// measured at a quarter of the L2 gather rate; pushing costs one remote store
// per entry and block and needs no answer.)
//
// Arithmetic: each segment is summed by the same lanes in the same order as in
// the task engine (kBatch FMA chains per lane, the lane group's shuffle tree),
// and every element update is the same expression, so iterates agree with the
// other forms up to the order of the compensated norms, whose FP64 totals
// differ in the last bits at most.
//
// What bounds it: with one or two passes per warp the chains of dependent
// instructions (cycle counters around each phase, 2,000 x 5,000 LP on 16 blocks,
// 14,100 cycles a step then, 12,400 now: the x' phase 1,050, its barrier with the average
// updates 2,100, A x' 2,200, barrier 1,150, A^T y' 3,250, barrier 1,400, the controller
// 2,550, of which one FP64 division 550 and a dozen dependent FP64 operations of
// 65 each); with four and more the number of instructions as well.  Microseconds
// per step, k_solo_steps (task engine for the batches) and here: 317 x 803 13.7 and
// 4.3, 2,000 x 5,000 13.7 and 6.4 (on 8 blocks 9.9), 64 of the latter as a batch 84 and
// 18.7 (clusters of four blocks, two rounds of them; with 16 bytes a pair of entries
// 43).  1, 2, 4 and 8 blocks for 317 x 803: 8.7, 6.6, 5.2 and 5.2 in an earlier state.  Why 16
// warps with passes at most: with 20 the batch 10 %, with 26, 30 or 13 20 % more; why
// x' by a thread per column and a pass's rest by code of its length: fewer
// instructions, 3 to 10 % each.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "eval.cuh"
#include "gridsync.cuh"
#include "plain.h"
#include "resident.h"

namespace sihg {

namespace {

constexpr int kResThreads = 544;   // most threads of a block of a cluster: 16 warps with passes, the controller
constexpr int kResWarps = kResThreads / 32;
constexpr int kGridThreads = 768;  // threads of a block of the grid form
constexpr int kColWords = 8;       // per column: x, K^T y (2), c, l, u, average (2); x' is in the copy
constexpr int kRowWords = 7;       // per row: y, K x (2), rl, ru, average (2); y' is in the copy
constexpr int kGridColWords = 5;   // over every SM: K^T y (2), c, average (2); the rest is in the column's record
constexpr int kGridRowWords = 6;   // K x (2), rl, ru, average (2); y and y' are in global memory
constexpr int kPlainColWords = 6;  // plain algorithm, per column: x, c, l, u, tau, best x
constexpr int kPlainRowWords = 4;  // per row: y, rl, ru, sigma

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The cluster barrier in two halves, so that work on a block's own data fits
// between them.
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Shared-window address of `p` in block `rank` of the cluster.
__device__ __forceinline__ unsigned map_rank(const void* p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void st_rank(unsigned addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

__device__ __forceinline__ void st_rank2(unsigned addr, float a, float b) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

// Stores v at *p in every block of the cluster; the lanes of a segment's group
// share the blocks.
__device__ __forceinline__ void push(float* p, float v, int sub, int L, int cluster) {
    if (cluster == 1) {
        if (sub == 0) *p = v;
        return;
    }
#pragma unroll 4
    for (int r = sub; r < cluster; r += L) st_rank(map_rank(p, r), v);
}

// Entries of a side: a lane's entries of a pass two at a time, 32 lanes together.
// In a cluster indices have 16 bits (its vectors fit in shared memory): 12
// bytes a pair instead of 16, a quarter less of what decides how many blocks
// an LP needs.  Empty places hold value 0 and the index of a zero behind the
// gathered vector, so that no lane has to ask.
struct Compact {
    static constexpr int kPair = 32 * 12;
    static __device__ __forceinline__ void load(const char* p, int& i0, float& a0, int& i1, float& a1) {
        const int lane = threadIdx.x & 31;
        const float2 a = *reinterpret_cast<const float2*>(p + 8 * lane);
        const unsigned i = *reinterpret_cast<const unsigned*>(p + 256 + 4 * lane);
        i0 = i & 0xffffu;
        i1 = i >> 16;
        a0 = a.x;
        a1 = a.y;
    }
    static __device__ __forceinline__ void store(char* p, int i0, float a0, int i1, float a1) {
        const int lane = threadIdx.x & 31;
        *reinterpret_cast<float2*>(p + 8 * lane) = make_float2(a0, a1);
        *reinterpret_cast<unsigned*>(p + 256 + 4 * lane) = (unsigned)i0 | (unsigned)i1 << 16;
    }
};
// Over every SM: 32-bit indices, empty places -1.
struct Wide {
    static constexpr int kPair = 32 * 16;
    static __device__ __forceinline__ void load(const char* p, int& i0, float& a0, int& i1, float& a1) {
        const int4 q = *reinterpret_cast<const int4*>(p + 16 * (threadIdx.x & 31));
        i0 = q.x;
        a0 = __int_as_float(q.y);
        i1 = q.z;
        a1 = __int_as_float(q.w);
    }
    static __device__ __forceinline__ void store(char* p, int i0, float a0, int i1, float a1) {
        *reinterpret_cast<int4*>(p + 16 * (threadIdx.x & 31)) =
            make_int4(i0, __float_as_int(a0), i1, __float_as_int(a1));
    }
};

// Gathers from a copy in shared memory; `none`: the index of the zero behind it.
struct FromShared {
    using Entries = Compact;
    const float* v;
    int none;
    __device__ __forceinline__ float operator()(int i) const { return v[i]; }
};

// Gathers of a vector written earlier in the same launch (coherent loads).
struct FromGlobal {
    using Entries = Wide;
    const float* v;
    __device__ __forceinline__ float operator()(int i) const {
        float x = 0.f;
        if (i >= 0) asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(v + i));
        return x;
    }
};

// The candidate x' of a column from its record {x, c + K^T y, l, u}.
__device__ __forceinline__ float x_from_record(const float4& r, float tau) {
    return fminf(fmaxf(fmaf(-tau, r.y, r.x), r.z), r.w);
}
__device__ __forceinline__ float4 ld_record(const float4* p) {
    float4 r;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
    return r;
}
struct FromRecords {
    using Entries = Wide;
    const float4* v;
    float tau;
    __device__ __forceinline__ float operator()(int i) const {
        return i >= 0 ? x_from_record(ld_record(v + i), tau) : 0.f;
    }
};

// Dot products of one pass: lane (group, sub) sums its entries with the values
// gather(index); the sum s + e (e: the compensation) is valid in each group's
// first lane.  The phases are bound by the latency and the number of these
// instructions, not by shared-memory bandwidth: four pairs of entries are read
// before the first is summed, and the rest of a pass by code of its length.
template <bool COMP, int PAIRS, class Gather>
__device__ __forceinline__ void sum_pairs(const char* rows, const Gather& gather, float (&acc)[kBatch], float& s,
                                          float& e) {
    using Entries = typename Gather::Entries;
    int i[2 * PAIRS];
    float a[2 * PAIRS], g[2 * PAIRS];
#pragma unroll
    for (int u = 0; u < PAIRS; ++u)
        Entries::load(rows + u * Entries::kPair, i[2 * u], a[2 * u], i[2 * u + 1], a[2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2 * PAIRS; ++u) g[u] = gather(i[u]);
#pragma unroll
    for (int u = 0; u < 2 * PAIRS; ++u) {
        if (COMP) {
            float pr, pe, ss, se;
            two_prod(a[u], g[u], pr, pe);
            two_sum(s, pr, ss, se);
            s = ss;
            e = __fadd_rn(e, __fadd_rn(pe, se));
        } else {
            acc[u % kBatch] = fmaf(a[u], g[u], acc[u % kBatch]);
        }
    }
}

template <bool COMP, class Gather>
__device__ __forceinline__ void pass_sums(const char* rows, int width, int lg, const Gather& gather, float& s,
                                          float& e) {
    float acc[kBatch] = {0.f, 0.f, 0.f, 0.f};
    s = e = 0.f;
    int pairs = (width + 1) >> 1;
    for (; pairs > 4; pairs -= 4, rows += 4 * Gather::Entries::kPair) sum_pairs<COMP, 4>(rows, gather, acc, s, e);
    if (pairs > 2) {
        if (pairs == 4)
            sum_pairs<COMP, 4>(rows, gather, acc, s, e);
        else
            sum_pairs<COMP, 3>(rows, gather, acc, s, e);
    } else if (pairs == 2) {
        sum_pairs<COMP, 2>(rows, gather, acc, s, e);
    } else if (pairs == 1) {
        sum_pairs<COMP, 1>(rows, gather, acc, s, e);
    }
    if (!COMP) s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    // the group's tree (the group's first lane adds as group_sum / group_sum2 do)
    for (int o = (1 << lg) >> 1; o > 0; o >>= 1) {
        const float s2 = __shfl_xor_sync(FULL_MASK, s, o);
        if (COMP) {
            const float e2 = __shfl_xor_sync(FULL_MASK, e, o);
            float t, te;
            two_sum(s, s2, t, te);
            s = t;
            e = __fadd_rn(e, __fadd_rn(e2, te));
        } else {
            s += s2;
        }
    }
}

// The same rounded to float, in every lane of the group.
template <bool COMP, class Gather>
__device__ __forceinline__ float pass_dot(const char* rows, int width, int lg, const Gather& gather) {
    float s, e;
    pass_sums<COMP>(rows, width, lg, gather, s, e);
    if (!COMP) return s;
    return __shfl_sync(FULL_MASK, __fadd_rn(s, e), (threadIdx.x & 31) >> lg << lg);
}

// What a step needs of the controller's state (FP32), published to the block.
struct StepPub {
    int cur, avg, done;
    float w, tau, sigma;
};

// One pass as a warp sees it: the segment of this lane's group.
template <class Entries>
struct PassOf {
    const char* rows;
    int width, lg, sub, seg, local;  // seg: in the instance, local: in the block
    bool on;                         // the group has a segment
    __device__ __forceinline__ PassOf(const int4& t, const char* side_rows) {
        const int lane = threadIdx.x & 31;
        rows = side_rows + t.x * Entries::kPair;
        width = t.y & 0xffffff;
        lg = t.y >> 24;
        const int g = lane >> lg;
        sub = lane & ((1 << lg) - 1);
        seg = t.z + g;
        local = (t.w & 0xffffff) + g;
        on = g < (t.w >> 24);
    }
};

using Pass = PassOf<Compact>;
using GridPass = PassOf<Wide>;

// Copies this block's passes and entries of both sides to shared memory.
template <class Entries>
__device__ __forceinline__ void load_block(const ResArgs& A, const ResBlock& blk, char* sm) {
    for (int h = 0; h < 2; ++h) {
        const ResSide& sd = blk.side[h];
        int4* pass = reinterpret_cast<int4*>(sm + A.sm.pass[h]);
        for (int k = threadIdx.x; k < sd.passes; k += blockDim.x) pass[k] = A.passes[sd.pass_begin + k];
        const int4* src = reinterpret_cast<const int4*>(A.rows + (size_t)sd.row_begin * Entries::kPair);
        int4* dst = reinterpret_cast<int4*>(sm + A.sm.rows[h]);
        for (int k = threadIdx.x; k < sd.rows * (Entries::kPair / 16); k += blockDim.x) dst[k] = __ldg(src + k);
    }
}

// Rows: K x' and the dual update (the operations of DualStepEpi::apply).
template <bool COMP>
__device__ __forceinline__ void dual_phase(const int4* pass, int passes, const char* rows, float* R, int nl, int cur,
                                           const FromShared& xs, float* ys, float sigma, int cluster, Acc& dy2) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const Pass t(pass[p], rows);
        const float kxp = pass_dot<COMP>(t.rows, t.width, t.lg, xs);
        if (t.on) {
            const float* r = R + t.local;
            const float yo = r[0], kx = r[(1 + cur) * nl], rl = r[3 * nl], ru = r[4 * nl];
            const float wv = (2.0f * kxp - kx) + yo / sigma;
            const float yv = sigma * (wv - fminf(fmaxf(wv, rl), ru));
            push(ys + t.seg, yv, t.sub, 1 << t.lg, cluster);
            if (t.sub == 0) {
                R[(1 + (cur ^ 1)) * nl + t.local] = kxp;
                const float dy = yv - yo;
                dy2.add(dy * dy);
            }
        }
    }
}

// Columns: K^T y', interaction and movement (the operations of KtyStepEpi::apply).
template <bool COMP>
__device__ __forceinline__ void kty_phase(const int4* pass, int passes, const char* rows, float* C, int nl, int cur,
                                          const FromShared& ys, const float* xs, Acc& inter, Acc& dx2) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const Pass t(pass[p], rows);
        const float k = pass_dot<COMP>(t.rows, t.width, t.lg, ys);
        if (t.on && t.sub == 0) {
            float* c = C + t.local;
            const float dx = xs[t.seg] - c[0];
            c[(1 + (cur ^ 1)) * nl] = k;
            inter.add(dx * (k - c[(1 + cur) * nl]));
            dx2.add(dx * dx);
        }
    }
}

// Sums a, b and c over the warp: a and b share one butterfly (the halves of
// the warp swap first: the lower lanes end with the total of a, the upper ones
// with that of b, both in `a`), c has its own beside it.
__device__ __forceinline__ void warp_reduce_three(Acc& a, Acc& b, Acc& c) {
    const bool up = (threadIdx.x & 16) != 0;
    Acc keep = up ? b : a, give = up ? a : b, got;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        got.s = __shfl_xor_sync(FULL_MASK, o == 16 ? give.s : keep.s, o);
        got.c = __shfl_xor_sync(FULL_MASK, o == 16 ? give.c : keep.c, o);
        keep = acc_plus(keep, got);
        got.s = __shfl_xor_sync(FULL_MASK, c.s, o);
        got.c = __shfl_xor_sync(FULL_MASK, c.c, o);
        c = acc_plus(c, got);
    }
    a = keep;
}

// The partial sums {inter, |dx|^2, |dy|^2} of a warp or a block.
struct Sums {
    float2 inter, dx2, dy2;
};

// Loads n (at most 32) of them, one per lane, and sums them over the warp (as
// warp_reduce_three).
__device__ __forceinline__ void reduce_sums(const Sums* p, int n, Acc& a, Acc& c) {
    const int lane = threadIdx.x & 31;
    Acc b;
    a.reset();
    c.reset();
    if (lane < n) {
        a.s = p[lane].inter.x;
        a.c = p[lane].inter.y;
        b.s = p[lane].dx2.x;
        b.c = p[lane].dx2.y;
        c.s = p[lane].dy2.x;
        c.c = p[lane].dy2.y;
    }
    warp_reduce_three(a, b, c);
}
// The step controller (step_controller), spread over the lanes of one warp.
// FP64 is slow here (65 cycles an addition or multiplication, 550 a division):
// what does not need the step's sums is prepared beside the A^T y' phase, and
// what does is one chain with one division, a lane each for eta_bar, the next
// eta and its tau and sigma.
struct StepCtrl {
    double coef, grow, om, inv_om, eta, W1, avg_w, dy2;
    bool nan, accept;

    __device__ __forceinline__ void prepare(const Inst& S) {
        const int lane = threadIdx.x & 31;
        om = S.omega;
        eta = S.eta;
        W1 = S.W + eta;
        const double quot = (lane == 1 ? eta : 1.0) / (lane == 1 ? W1 : om);
        inv_om = __shfl_sync(FULL_MASK, quot, 0);
        avg_w = __shfl_sync(FULL_MASK, quot, 1);
        const double per = lane == 2 ? inv_om : (lane == 3 ? om : 1.0);
        grow = (1.0 + S.pow06) * eta * per;
        coef = lane == 0 ? 1.0 : (1.0 - S.pow03) * per;
    }
    // From n partial sums of the step.
    __device__ __forceinline__ void decide(const Sums* sums, int n, StepPub& pub) {
        const int lane = threadIdx.x & 31;
        Acc two, d;
        reduce_sums(sums, n, two, d);
        const double mine = (double)two.s + (double)two.c;
        dy2 = (double)d.s + (double)d.c;
        const double inter = __shfl_sync(FULL_MASK, mine, 0), dx2 = __shfl_sync(FULL_MASK, mine, 16);
        // lane 0 eta_bar, lane 1 (1 - k^-0.3) eta_bar, lanes 2 and 3 the same
        // / and * omega.  Non-negative FP64 numbers compare as integers (FP64
        // compares have the latency of FP64 sums); a NaN compares above infinity.
        const double movement = om * dx2 + dy2 * inv_om;
        const double ai = fabs(inter);
        const double quot = __double_as_longlong(ai) != 0 ? coef * movement / (2.0 * ai) : INFINITY;
        const long long qb = __double_as_longlong(quot), inf = 0x7ff0000000000000ll;
        const bool less = __shfl_sync(FULL_MASK, (int)(qb < __double_as_longlong(grow)), 1) != 0;
        const double next = less ? quot : grow;
        nan = __double_as_longlong(fabs(movement)) > inf || __double_as_longlong(ai) > inf;
        accept = !nan && __double_as_longlong(eta) <= qb && qb <= inf;  // lane 0
        if (nan) {
            if (lane == 0) pub.done = 3;
            return;
        }
        if (lane == 2) pub.tau = (float)next;
        if (lane == 3) pub.sigma = (float)next;
        if (lane == 0) {
            pub.avg = accept;
            if (accept) {
                pub.cur ^= 1;
                pub.w = (float)avg_w;
            }
        }
        eta = __shfl_sync(FULL_MASK, next, 1);
    }
    // The instance's state after the step (lane 0, beside the next phase).
    __device__ __forceinline__ void record(Inst& S) const {
        S.attempts += 1;
        if (nan) {
            S.done = 3;
            return;
        }
        S.dy2 = dy2;
        S.avg_pending = accept;
        if (accept) {
            S.cur ^= 1;
            S.steps += 1;
            S.since_restart += 1;
            S.W = W1;
            S.avg_w = avg_w;
        } else {
            S.rejections += 1;
        }
        S.eta = eta;
    }
};

constexpr int kEvalQ = 18;  // reductions of an evaluation: 8 of the rows, 10 of the columns

// Sums of a side's segments with the first candidate point, to s and e by local segment.
__device__ __forceinline__ void eval_sums(bool comp, const int4* pass, int passes, const char* rows, const FromShared& vec,
                                          float* s_out, float* e_out) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const Pass t(pass[p], rows);
        float s, e;
        if (comp)
            pass_sums<true>(t.rows, t.width, t.lg, vec, s, e);
        else
            pass_sums<false>(t.rows, t.width, t.lg, vec, s, e);
        if (t.on && t.sub == 0) {
            s_out[t.local] = s;
            e_out[t.local] = e;
        }
    }
}

// The evaluation epilogue of a side's segments: first candidate's sums from s
// and e, the second's from `vec`; `first` is the instance's first segment.
template <class Epi>
__device__ __forceinline__ void eval_apply(bool comp, const int4* pass, int passes, const char* rows, const FromShared& vec,
                                           const float* s_in, const float* e_in, int first, Epi& epi) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const Pass t(pass[p], rows);
        SegDot<2> d;
        if (comp)
            pass_sums<true>(t.rows, t.width, t.lg, vec, d.s[1], d.e[1]);
        else
            pass_sums<false>(t.rows, t.width, t.lg, vec, d.s[1], d.e[1]);
        if (t.on && t.sub == 0) {
            d.s[0] = s_in[t.local];
            d.e[0] = e_in[t.local];
            epi.apply(first + t.seg, d, epi.pre(first + t.seg));
        }
    }
}

// Total of n (at most 32) partials of reduction i, in every lane.
__device__ __forceinline__ Acc eval_total(const float2* p, int n, int i) {
    const int lane = threadIdx.x & 31;
    Acc v[1];
    if (lane < n) {
        v[0].s = p[lane].x;
        v[0].c = p[lane].y;
    }
    const bool is_max = i == 2 || i == 3 || i == 10 || i == 11;
    warp_reduce_acc<1>(v, is_max ? 1u : 0u);
    return v[0];
}

}  // namespace

// Blocks: all warps but the last own passes; the last warp runs the step
// controller (every block its own copy, from the same partials, so that no
// answer has to come back).
__global__ void __launch_bounds__(kResThreads, 1) k_resident_steps(ResArgs A, int nsteps, int periods, Vecs V, Inst* st, unsigned* done_count) {
    extern __shared__ char sm[];
    __shared__ Inst S;  // the controller's copy (its first lane's)
    __shared__ StepPub pub;
    __shared__ int flag;
    __shared__ unsigned ignored;  // done count of the other blocks' controller copies
    const int inst = blockIdx.x / A.cluster, cluster = A.cluster;
    if (st[inst].done) return;  // the whole cluster
    const int rank = cluster > 1 ? (int)cluster_rank() : 0;
    const ResBlock& blk = A.blocks[blockIdx.x];
    const int4 io = A.inst[inst];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x >> 5) - 1;
    const bool ctrl = warp == nw;
    int4* rpass = reinterpret_cast<int4*>(sm + A.sm.pass[0]);
    int4* cpass = reinterpret_cast<int4*>(sm + A.sm.pass[1]);
    const char* rrows = sm + A.sm.rows[0];
    const char* crows = sm + A.sm.rows[1];
    float* xs = reinterpret_cast<float*>(sm + A.sm.xs);
    float* ys = reinterpret_cast<float*>(sm + A.sm.ys);
    float* C = reinterpret_cast<float*>(sm + A.sm.col);  // x | K^T y, K^T y' | c l u | average hi lo
    float* R = reinterpret_cast<float*>(sm + A.sm.row);  // y | K x, K x' | rl ru | average hi lo
    Sums* wsum = reinterpret_cast<Sums*>(sm + A.sm.red);  // of every warp of this block
    Sums* bsum = wsum + kResWarps;                        // of every block of the cluster
    unsigned short* cseg = reinterpret_cast<unsigned short*>(sm + A.sm.seg);  // segment of each local column
    const int ncl = A.sm.locals[1], nrl = A.sm.locals[0];
    const int rp = blk.side[0].passes, cp = blk.side[1].passes, nc = blk.side[1].locals;
    const FromShared gx{xs, io.y}, gy{ys, io.w};
    if (threadIdx.x == 0) xs[io.y] = ys[io.w] = 0.f;
    load_block<Compact>(A, blk, sm);
    if (threadIdx.x == 0) {
        S = st[inst];
        const StepScalars sc = step_scalars(S);
        pub = StepPub{sc.cur, sc.avg, 0, sc.w, sc.tau, (float)(S.eta * S.omega)};
    }
    __syncthreads();
    if (!ctrl) {  // owners' data
        const int cur = pub.cur;
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            if (t.on && t.sub == 0) {
                const int j = io.x + t.seg;
                float* c = C + t.local;
                cseg[t.local] = (unsigned short)t.seg;
                xs[t.seg] = c[0] = pick(V.x0, V.x1, cur)[j];
                c[(1 + cur) * ncl] = pick(V.kty0, V.kty1, cur)[j];
                c[3 * ncl] = V.c[j];
                c[4 * ncl] = V.l[j];
                c[5 * ncl] = V.u[j];
                const float2 a = V.x_acc[j];
                c[6 * ncl] = a.x;
                c[7 * ncl] = a.y;
            }
        }
        for (int p = warp; p < rp; p += nw) {
            const Pass t(rpass[p], rrows);
            if (t.on && t.sub == 0) {
                const int j = io.z + t.seg;
                float* r = R + t.local;
                ys[t.seg] = r[0] = pick(V.y0, V.y1, cur)[j];
                r[(1 + cur) * nrl] = pick(V.kx0, V.kx1, cur)[j];
                r[3 * nrl] = V.rl[j];
                r[4 * nrl] = V.ru[j];
                const float2 a = V.y_acc[j];
                r[5 * nrl] = a.x;
                r[6 * nrl] = a.y;
            }
        }
    }
    cluster_arrive();  // every block of the cluster runs before the first remote store
    cluster_wait();
    for (int period = 0; period < periods && !pub.done; ++period) {
    const bool comp = S.refine != 0;
    for (int k = 0; k < nsteps && !pub.done; ++k) {
        const int cur = pub.cur;
        const bool avg = pub.avg != 0;
        const float w = pub.w, tau = pub.tau, sg = pub.sigma;
        // x' = clip(x - tau (c + K^T y), l, u); after an accepted step x is the
        // candidate of that step, still in the copy
        if (!ctrl) {
            for (int l = threadIdx.x; l < nc; l += 32 * nw) {
                float* c = C + l;
                const int seg = cseg[l];
                const float x = avg ? xs[seg] : c[0];
                const float v = fmaf(-tau, c[3 * ncl] + c[(1 + cur) * ncl], x);
                push(xs + seg, fminf(fmaxf(v, c[4 * ncl]), c[5 * ncl]), 0, 1, cluster);
                c[0] = x;
            }
        }
        cluster_arrive();
        if (ctrl) {
            if (lane == 0) schedule_pows(S, V);
        } else if (avg) {  // the pending average updates, while the other blocks arrive
            for (int l = threadIdx.x; l < nc; l += 32 * nw) {
                float* c = C + l;
                const float2 a = ff_axpy(make_float2(c[6 * ncl], c[7 * ncl]), w, c[0]);
                c[6 * ncl] = a.x;
                c[7 * ncl] = a.y;
            }
            for (int p = warp; p < rp; p += nw) {
                const Pass t(rpass[p], rrows);
                if (t.on && t.sub == 0) {
                    float* r = R + t.local;
                    const float y = r[0] = ys[t.seg];
                    const float2 a = ff_axpy(make_float2(r[5 * nrl], r[6 * nrl]), w, y);
                    r[5 * nrl] = a.x;
                    r[6 * nrl] = a.y;
                }
            }
            __syncwarp();  // the whole group reads y in the next phase
        }
        cluster_wait();
        Acc dy2;
        if (!ctrl) {
            if (comp)
                dual_phase<true>(rpass, rp, rrows, R, nrl, cur, gx, ys, sg, cluster, dy2);
            else
                dual_phase<false>(rpass, rp, rrows, R, nrl, cur, gx, ys, sg, cluster, dy2);
        }
        cluster_arrive();
        cluster_wait();
        StepCtrl ctl;
        if (!ctrl) {
            Acc inter, dx2;
            if (comp)
                kty_phase<true>(cpass, cp, crows, C, ncl, cur, gy, xs, inter, dx2);
            else
                kty_phase<false>(cpass, cp, crows, C, ncl, cur, gy, xs, inter, dx2);
            warp_reduce_three(inter, dx2, dy2);  // inter: |dx|^2 in the upper lanes
            if (lane == 0) {
                wsum[warp].inter = make_float2(inter.s, inter.c);
                wsum[warp].dy2 = make_float2(dy2.s, dy2.c);
            }
            if (lane == 16) wsum[warp].dx2 = make_float2(inter.s, inter.c);
        } else {
            ctl.prepare(S);
        }
        __syncthreads();
        if (ctrl) {  // the block's sums to every block: lane r (inter, |dy|^2) and 16 + r (|dx|^2) to block r
            Acc a, c;
            reduce_sums(wsum, nw, a, c);
            if ((lane & 15) < cluster) {
                st_rank2(map_rank(lane < 16 ? &bsum[rank].inter : &bsum[rank].dx2, lane & 15), a.s, a.c);
                if (lane < 16) st_rank2(map_rank(&bsum[rank].dy2, lane), c.s, c.c);
            }
        }
        cluster_arrive();
        cluster_wait();
        if (ctrl) ctl.decide(bsum, cluster, pub);
        __syncthreads();
        if (ctrl && lane == 0) ctl.record(S);
    }
    // The evaluation (as k_flush_avg, k_eval_rows, k_eval_cols and k_restart):
    // the copies hold the current point, then the average one; the epilogues
    // read their segments' data from global memory, where the owners put the
    // current point first.
    const int cur = pub.cur;
    const bool avg = pub.avg != 0;
    const bool failed = pub.done != 0;  // a step of this period: nothing to evaluate, and no store to a block that may have ended
    const float w = pub.w;
    if (!ctrl) {
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            float x = 0.f;
            if (t.on) x = avg ? xs[t.seg] : C[t.local];
            __syncwarp();
            if (t.on) {
                if (!failed) push(xs + t.seg, x, t.sub, 1 << t.lg, cluster);
                if (t.sub == 0) {
                    const int j = io.x + t.seg;
                    float* c = C + t.local;
                    float2 a = make_float2(c[6 * ncl], c[7 * ncl]);
                    if (avg) a = ff_axpy(a, w, x);
                    c[6 * ncl] = a.x;
                    c[7 * ncl] = a.y;
                    pick(V.x0, V.x1, cur)[j] = x;
                    pick(V.kty0, V.kty1, cur)[j] = c[(1 + cur) * ncl];
                    V.x_acc[j] = a;
                    V.x_avg[j] = __fadd_rn(a.x, a.y);
                }
            }
        }
        for (int p = warp; p < rp; p += nw) {
            const Pass t(rpass[p], rrows);
            float y = 0.f;
            if (t.on) y = avg ? ys[t.seg] : R[t.local];
            __syncwarp();
            if (t.on) {
                if (!failed) push(ys + t.seg, y, t.sub, 1 << t.lg, cluster);
                if (t.sub == 0) {
                    const int j = io.z + t.seg;
                    float* r = R + t.local;
                    float2 a = make_float2(r[5 * nrl], r[6 * nrl]);
                    if (avg) a = ff_axpy(a, w, y);
                    r[5 * nrl] = a.x;
                    r[6 * nrl] = a.y;
                    pick(V.y0, V.y1, cur)[j] = y;
                    pick(V.kx0, V.kx1, cur)[j] = r[(1 + cur) * nrl];
                    V.y_acc[j] = a;
                    V.y_avg[j] = __fadd_rn(a.x, a.y);
                }
            }
        }
        __syncwarp();  // the groups read the averages below
    }
    if (failed) {
        if (rank == 0 && ctrl && lane == 0) st[inst] = S;
        return;
    }
    cluster_arrive();
    cluster_wait();
    if (!ctrl) {  // the current point's sums, kept where the point (now in global memory) and the candidate's product were
        eval_sums(comp, rpass, rp, rrows, gx, R, R + (1 + (cur ^ 1)) * nrl);
        eval_sums(comp, cpass, cp, crows, gy, C, C + (1 + (cur ^ 1)) * ncl);
    }
    cluster_arrive();
    cluster_wait();
    if (!ctrl) {
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            if (t.on)
                push(xs + t.seg, __fadd_rn(C[6 * ncl + t.local], C[7 * ncl + t.local]), t.sub, 1 << t.lg, cluster);
        }
        for (int p = warp; p < rp; p += nw) {
            const Pass t(rpass[p], rrows);
            if (t.on)
                push(ys + t.seg, __fadd_rn(R[5 * nrl + t.local], R[6 * nrl + t.local]), t.sub, 1 << t.lg, cluster);
        }
    }
    cluster_arrive();
    cluster_wait();
    float2* ewarp = reinterpret_cast<float2*>(sm + A.sm.eval);  // [kEvalQ][kResWarps] of the block's warps
    float2* eblock = ewarp + kEvalQ * kResWarps;                // [kEvalQ][16] of the cluster's blocks
    double* etot = reinterpret_cast<double*>(eblock + kEvalQ * 16);
    if (!ctrl) {
        EvalRowsEpi er{V};
        er.begin(S);
        Acc q[8];
        eval_apply(comp, rpass, rp, rrows, gx, R, R + (1 + (cur ^ 1)) * nrl, io.z, er);
        er.values(q);
        warp_reduce_acc<8>(q, 0x0Cu);
        if (lane == 0)
            for (int i = 0; i < 8; ++i) ewarp[i * kResWarps + warp] = make_float2(q[i].s, q[i].c);
    }
    if (!ctrl) {
        EvalColsEpi ec{V, nullptr};
        ec.begin(S);
        Acc q[10];
        eval_apply(comp, cpass, cp, crows, gy, C, C + (1 + (cur ^ 1)) * ncl, io.x, ec);
        ec.values(q);
        warp_reduce_acc<10>(q, 0x0Cu);
        if (lane == 0)
            for (int i = 0; i < 10; ++i) ewarp[(8 + i) * kResWarps + warp] = make_float2(q[i].s, q[i].c);
    }
    __syncthreads();
    for (int i = warp; i < kEvalQ; i += nw + 1) {
        const Acc v = eval_total(ewarp + i * kResWarps, nw, i);
        if (lane < cluster) st_rank2(map_rank(eblock + i * 16 + rank, lane), v.s, v.c);
    }
    cluster_arrive();
    cluster_wait();
    for (int i = warp; i < kEvalQ; i += nw + 1) {
        const Acc v = eval_total(eblock + i * 16, cluster, i);
        if (lane == 0) etot[i] = (double)v.s + (double)v.c;
    }
    __syncthreads();
    if (ctrl && lane == 0) {
        for (int i = 0; i < 8; ++i) S.row_eval[i] = etot[i];
        S.col_eval_dist[0] = etot[16];
        S.col_eval_dist[1] = etot[17];
        eval_controller(S, etot + 8, rank == 0 ? done_count : &ignored);
        const StepScalars sc = step_scalars(S);
        pub = StepPub{sc.cur, 0, S.done, sc.w, sc.tau, (float)(S.eta * S.omega)};
        flag = S.restart_flag;
    }
    __syncthreads();
    if (!ctrl) {  // the point back, after a restart at the current (1) or the average point (2) with its average
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            if (t.on && t.sub == 0) {
                const int j = io.x + t.seg;
                float* c = C + t.local;
                float* gx0 = pick(V.x0, V.x1, cur) + j;
                if (flag == 2) {
                    *gx0 = V.x_avg[j];
                    pick(V.kty0, V.kty1, cur)[j] = c[(1 + cur) * ncl] = V.kty_eval[j];
                }
                const float x = c[0] = *gx0;
                if (flag != 0) {
                    V.x_last[j] = x;
                    V.x_acc[j] = make_float2(x, 0.f);
                    c[6 * ncl] = x;
                    c[7 * ncl] = 0.f;
                }
            }
        }
        for (int p = warp; p < rp; p += nw) {
            const Pass t(rpass[p], rrows);
            if (t.on && t.sub == 0) {
                const int j = io.z + t.seg;
                float* r = R + t.local;
                float* gy0 = pick(V.y0, V.y1, cur) + j;
                if (flag == 2) {
                    *gy0 = V.y_avg[j];
                    pick(V.kx0, V.kx1, cur)[j] = r[(1 + cur) * nrl] = V.kx_eval[j];
                }
                const float y = r[0] = *gy0;
                if (flag != 0) {
                    V.y_last[j] = y;
                    V.y_acc[j] = make_float2(y, 0.f);
                    r[5 * nrl] = y;
                    r[6 * nrl] = 0.f;
                }
            }
        }
    }
    __syncthreads();  // other threads read x and y in the next step
    }
    if (rank == 0 && ctrl && lane == 0) st[inst] = S;
}

// ---------------------------------------------------------------- grid form
// One LP over every SM: the same layout with a block per SM instead of a block
// of a cluster.  The matrix and the owners' data stay in shared memory; x' and
// y' are gathered from L2 (x' computed by the gathering lane from its column's
// record, so that a step needs two grid barriers), and the barrier after
// A^T y' carries the blocks' sums.
//
// What bounds it (cycle counters, refinery LP with 24 / 168 periods, 18,000 /
// 28,800 cycles a step): A x' 2,300 / 6,400, its barrier 4,400 / 4,900, A^T y' 2,900 /
// 8,200, the block's sums 700, the second barrier 3,300, the grid's sums 1,300,
// the controller 2,300.  The small LP is barriers (a release, an L2 round trip and
// an acquire each) and the controller's FP64 chain; the large one as much the
// instructions of its 50 passes a side and block (about 300 each, compensated
// sums near the tolerance).  Measured per step, whole solves: 14.6 -> 9.0 us and
// 26 -> 14.4 us against k_solo_steps, which reads the matrix from L2 (LPs that do
// not fit step over packs, see kPackMinNnz); with the rest of a pass by code of
// its length, steps alone, 8.75 -> 8.6 and 13.8 -> 12.9 us.
//
// Grid-wide barrier.  Every block adds one to its counter of kArrive (fewer
// additions queue up at one address) with release semantics; one warp of each
// block polls all of them with relaxed loads, then acquires once (an acquire
// per poll, or a flag per block polled by a thread each, took 5,600 - 7,300
// cycles a barrier).  Waits are bounded as in gridsync.cuh; false: give up.
constexpr int kArrive = 8;
struct GridSync {
    unsigned* count;  // [kArrive] counters, 32 words apart, then `turn`; zeroed before a run
    int* status;
    unsigned long long limit_ns;
    unsigned turn;    // barriers passed

    __device__ __forceinline__ bool operator()(bool* ok) {
        ++turn;
        __syncthreads();
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            if (lane == 0)
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count + 32 * (blockIdx.x % kArrive))
                             : "memory");
            // blocks that share counter `lane`, times the barriers so far
            const unsigned mine = lane < kArrive ? (gridDim.x - lane + kArrive - 1) / kArrive * turn : 0u;
            const unsigned long long t0 = global_ns();
            unsigned spins = 0;
            bool good = true;
            for (;;) {
                unsigned v = mine;
                if (lane < kArrive)
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count + 32 * lane) : "memory");
                if (__all_sync(FULL_MASK, (int)(v - mine) >= 0)) break;
                if ((++spins & 31u) == 0u) {
                    const bool late = global_ns() - t0 > limit_ns;
                    if (lane == 0 && late) atomicExch(status, 1);
                    if (__any_sync(FULL_MASK, late || ld_status(status) != 0)) {
                        good = false;
                        break;
                    }
                }
            }
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            if (lane == 0) *ok = good;
        }
        __syncthreads();
        return *ok;
    }
};

// Columns of the grid form: K^T y' from L2, x' from the owner's record, the
// next record, and the average update (the operations of KtyStepEpiPacked).
template <bool COMP>
__device__ __forceinline__ void grid_cols(const int4* pass, int passes, const char* rows, float* C, int nl, int cur,
                                          const float* y, const float4* records, float4* next, float tau, bool avg,
                                          float w, Acc& inter, Acc& dx2) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const GridPass t(pass[p], rows);
        float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t.on && t.sub == 0) rec = ld_record(records + t.seg);
        const float k = pass_dot<COMP>(t.rows, t.width, t.lg, FromGlobal{y});
        if (t.on && t.sub == 0) {
            float* c = C + t.local;
            const float x = rec.x, kty = c[cur * nl], cc = c[2 * nl];
            const float xp = x_from_record(rec, tau);
            if (avg) {
                const float2 a = ff_axpy(make_float2(c[3 * nl], c[4 * nl]), w, x);
                c[3 * nl] = a.x;
                c[4 * nl] = a.y;
            }
            c[(cur ^ 1) * nl] = k;
            next[t.seg] = make_float4(xp, cc + k, rec.z, rec.w);
            const float dx = xp - x;
            inter.add(dx * (k - kty));
            dx2.add(dx * dx);
        }
    }
}

// Rows: K x' gathered through the records, dual update, average update.
template <bool COMP>
__device__ __forceinline__ void grid_rows(const int4* pass, int passes, const char* rows, float* R, int nl, int cur,
                                          const float4* records, float tau, float sigma, const float* y, float* y_next,
                                          bool avg, float w, Acc& dy2) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const GridPass t(pass[p], rows);
        float yo = 0.f;
        if (t.on && t.sub == 0) yo = FromGlobal{y}(t.seg);
        const float kxp = pass_dot<COMP>(t.rows, t.width, t.lg, FromRecords{records, tau});
        if (t.on && t.sub == 0) {
            float* r = R + t.local;
            const float kx = r[cur * nl], rl = r[2 * nl], ru = r[3 * nl];
            if (avg) {
                const float2 a = ff_axpy(make_float2(r[4 * nl], r[5 * nl]), w, yo);
                r[4 * nl] = a.x;
                r[5 * nl] = a.y;
            }
            const float wv = (2.0f * kxp - kx) + yo / sigma;
            const float yv = sigma * (wv - fminf(fmaxf(wv, rl), ru));
            r[(cur ^ 1) * nl] = kxp;
            y_next[t.seg] = yv;
            const float dy = yv - yo;
            dy2.add(dy * dy);
        }
    }
}

// The evaluation epilogue over a side, both candidates gathered from L2.
template <bool COMP, class Epi>
__device__ __forceinline__ void grid_eval(const int4* pass, int passes, const char* rows, const float* v0,
                                          const float* v1, Epi& epi) {
    const int nw = (blockDim.x >> 5) - 1;
    for (int p = threadIdx.x >> 5; p < passes; p += nw) {
        const GridPass t(pass[p], rows);
        SegDot<2> d;
        pass_sums<COMP>(t.rows, t.width, t.lg, FromGlobal{v0}, d.s[0], d.e[0]);
        pass_sums<COMP>(t.rows, t.width, t.lg, FromGlobal{v1}, d.s[1], d.e[1]);
        if (t.on && t.sub == 0) epi.apply(t.seg, d, epi.pre(t.seg));
    }
}

__global__ void __launch_bounds__(kGridThreads, 1)
    k_resident_grid(ResArgs A, int nsteps, int periods, Vecs V, Inst* st, unsigned* done_count, float4* records, int N,
                    unsigned* count, Sums* bsum, float2* esums, GridBar gb) {
    extern __shared__ char sm[];
    __shared__ Inst S;
    __shared__ StepPub pub;
    __shared__ int flag;
    __shared__ unsigned ignored;
    __shared__ bool ok;
    if (st->done || ld_status(gb.status) != 0) return;
    const ResBlock& blk = A.blocks[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x >> 5) - 1, P = gridDim.x;
    const bool ctrl = warp == nw;
    int4* rpass = reinterpret_cast<int4*>(sm + A.sm.pass[0]);
    int4* cpass = reinterpret_cast<int4*>(sm + A.sm.pass[1]);
    const char* rrows = sm + A.sm.rows[0];
    const char* crows = sm + A.sm.rows[1];
    float* C = reinterpret_cast<float*>(sm + A.sm.col);  // K^T y, K^T y' | c | average hi lo
    float* R = reinterpret_cast<float*>(sm + A.sm.row);  // K x, K x' | rl ru | average hi lo
    Sums* wsum = reinterpret_cast<Sums*>(sm + A.sm.red);
    float2* ewarp = reinterpret_cast<float2*>(sm + A.sm.eval);
    double* etot = reinterpret_cast<double*>(ewarp + kEvalQ * 32);
    const int ncl = A.sm.locals[1], nrl = A.sm.locals[0];
    const int rp = blk.side[0].passes, cp = blk.side[1].passes;
    GridSync sync{count, gb.status, gb.limit_ns, count[32 * kArrive]};  // barriers of this run's earlier launches
    load_block<Wide>(A, blk, sm);
    if (threadIdx.x == 0) {
        S = *st;
        const StepScalars sc = step_scalars(S);
        pub = StepPub{sc.cur, sc.avg, 0, sc.w, sc.tau, (float)(S.eta * S.omega)};
    }
    __syncthreads();
    if (!ctrl) {  // owners' data and the records of the current point
        const int cur = pub.cur;
        for (int p = warp; p < cp; p += nw) {
            const GridPass t(cpass[p], crows);
            if (t.on && t.sub == 0) {
                const int j = t.seg;
                float* c = C + t.local;
                const float kty = c[cur * ncl] = pick(V.kty0, V.kty1, cur)[j];
                const float cc = c[2 * ncl] = V.c[j];
                const float2 a = V.x_acc[j];
                c[3 * ncl] = a.x;
                c[4 * ncl] = a.y;
                records[(size_t)cur * N + j] = make_float4(pick(V.x0, V.x1, cur)[j], cc + kty, V.l[j], V.u[j]);
            }
        }
        for (int p = warp; p < rp; p += nw) {
            const GridPass t(rpass[p], rrows);
            if (t.on && t.sub == 0) {
                const int j = t.seg;
                float* r = R + t.local;
                r[cur * nrl] = pick(V.kx0, V.kx1, cur)[j];
                r[2 * nrl] = V.rl[j];
                r[3 * nrl] = V.ru[j];
                const float2 a = V.y_acc[j];
                r[4 * nrl] = a.x;
                r[5 * nrl] = a.y;
            }
        }
    }
    if (!sync(&ok)) return;
    for (int period = 0; period < periods && !pub.done; ++period) {
        const bool comp = S.refine != 0;
        for (int k = 0; k < nsteps && !pub.done; ++k) {
            const int cur = pub.cur;
            const bool avg = pub.avg != 0;
            const float w = pub.w, tau = pub.tau, sg = pub.sigma;
            const float4* rec = records + (size_t)cur * N;
            const float* yc = pick(V.y0, V.y1, cur);
            float* yn = pick(V.y0, V.y1, cur ^ 1);
            Acc inter, dx2, dy2;
            StepCtrl ctl;
            if (!ctrl) {
                if (comp)
                    grid_rows<true>(rpass, rp, rrows, R, nrl, cur, rec, tau, sg, yc, yn, avg, w, dy2);
                else
                    grid_rows<false>(rpass, rp, rrows, R, nrl, cur, rec, tau, sg, yc, yn, avg, w, dy2);
            } else if (lane == 0) {
                schedule_pows(S, V);
            }
            if (!sync(&ok)) return;
            if (!ctrl) {
                float4* next = records + (size_t)(cur ^ 1) * N;
                if (comp)
                    grid_cols<true>(cpass, cp, crows, C, ncl, cur, yn, rec, next, tau, avg, w, inter, dx2);
                else
                    grid_cols<false>(cpass, cp, crows, C, ncl, cur, yn, rec, next, tau, avg, w, inter, dx2);
                warp_reduce_three(inter, dx2, dy2);
                if (lane == 0) {
                    wsum[warp].inter = make_float2(inter.s, inter.c);
                    wsum[warp].dy2 = make_float2(dy2.s, dy2.c);
                }
                if (lane == 16) wsum[warp].dx2 = make_float2(inter.s, inter.c);
            } else {
                ctl.prepare(S);
            }
            __syncthreads();
            if (warp == 0) {
                Acc a, c;
                reduce_sums(wsum, nw, a, c);
                if (lane == 0) {
                    bsum[blockIdx.x].inter = make_float2(a.s, a.c);
                    bsum[blockIdx.x].dy2 = make_float2(c.s, c.c);
                }
                if (lane == 16) bsum[blockIdx.x].dx2 = make_float2(a.s, a.c);
                __syncwarp();
            }
            if (!sync(&ok)) return;
            // the blocks' sums: one per thread, five warps, then the controller
            // (overwritten only after the next barrier)
            const int sw = (P + 31) / 32;
            if (warp < sw) {
                Acc i1, i2, i3;
                if (threadIdx.x < P) {
                    const float2* f = &bsum[threadIdx.x].inter;
                    const float2 f1 = __ldcg(f), f2 = __ldcg(f + 1), f3 = __ldcg(f + 2);
                    i1.s = f1.x;
                    i1.c = f1.y;
                    i2.s = f2.x;
                    i2.c = f2.y;
                    i3.s = f3.x;
                    i3.c = f3.y;
                }
                warp_reduce_three(i1, i2, i3);
                if (lane == 0) {
                    wsum[warp].inter = make_float2(i1.s, i1.c);
                    wsum[warp].dy2 = make_float2(i3.s, i3.c);
                }
                if (lane == 16) wsum[warp].dx2 = make_float2(i1.s, i1.c);
            }
            __syncthreads();
            if (ctrl) ctl.decide(wsum, sw, pub);
            __syncthreads();
            if (ctrl && lane == 0) ctl.record(S);
        }
        // The evaluation (as k_flush_avg, k_eval_rows, k_eval_cols and k_restart).
        const int cur = pub.cur;
        const bool avg = pub.avg != 0;
        const float w = pub.w;
        if (!ctrl) {
            for (int p = warp; p < cp; p += nw) {
                const GridPass t(cpass[p], crows);
                if (t.on && t.sub == 0) {
                    const int j = t.seg;
                    float* c = C + t.local;
                    const float x = ld_record(records + (size_t)cur * N + j).x;
                    float2 a = make_float2(c[3 * ncl], c[4 * ncl]);
                    if (avg) a = ff_axpy(a, w, x);
                    c[3 * ncl] = a.x;
                    c[4 * ncl] = a.y;
                    pick(V.x0, V.x1, cur)[j] = x;
                    pick(V.kty0, V.kty1, cur)[j] = c[cur * ncl];
                    V.x_acc[j] = a;
                    V.x_avg[j] = __fadd_rn(a.x, a.y);
                }
            }
            for (int p = warp; p < rp; p += nw) {
                const GridPass t(rpass[p], rrows);
                if (t.on && t.sub == 0) {
                    const int j = t.seg;
                    float* r = R + t.local;
                    float2 a = make_float2(r[4 * nrl], r[5 * nrl]);
                    if (avg) a = ff_axpy(a, w, FromGlobal{pick(V.y0, V.y1, cur)}(j));
                    r[4 * nrl] = a.x;
                    r[5 * nrl] = a.y;
                    pick(V.kx0, V.kx1, cur)[j] = r[cur * nrl];
                    V.y_acc[j] = a;
                    V.y_avg[j] = __fadd_rn(a.x, a.y);
                }
            }
        }
        if (pub.done) break;  // a step failed: nothing to evaluate
        if (!sync(&ok)) return;
        if (!ctrl) {
            EvalRowsEpi er{V};
            er.begin(S);
            Acc q[8];
            if (comp)
                grid_eval<true>(rpass, rp, rrows, er.xg[0], er.xg[1], er);
            else
                grid_eval<false>(rpass, rp, rrows, er.xg[0], er.xg[1], er);
            er.values(q);
            warp_reduce_acc<8>(q, 0x0Cu);
            if (lane == 0)
                for (int i = 0; i < 8; ++i) ewarp[i * 32 + warp] = make_float2(q[i].s, q[i].c);
        }
        if (!ctrl) {
            EvalColsEpi ec{V, nullptr};
            ec.begin(S);
            Acc q[10];
            if (comp)
                grid_eval<true>(cpass, cp, crows, ec.yg[0], ec.yg[1], ec);
            else
                grid_eval<false>(cpass, cp, crows, ec.yg[0], ec.yg[1], ec);
            ec.values(q);
            warp_reduce_acc<10>(q, 0x0Cu);
            if (lane == 0)
                for (int i = 0; i < 10; ++i) ewarp[(8 + i) * 32 + warp] = make_float2(q[i].s, q[i].c);
        }
        __syncthreads();
        for (int i = warp; i < kEvalQ; i += nw + 1) {
            const Acc v = eval_total(ewarp + i * 32, nw, i);
            if (lane == 0) esums[(size_t)i * P + blockIdx.x] = make_float2(v.s, v.c);
        }
        if (!sync(&ok)) return;
        for (int i = warp; i < kEvalQ; i += nw + 1) {
            const bool is_max = i == 2 || i == 3 || i == 10 || i == 11;
            Acc v[1];
            for (int k = lane; k < P; k += 32) {
                const float2 f = __ldcg(esums + (size_t)i * P + k);
                Acc b;
                b.s = f.x;
                b.c = f.y;
                v[0] = acc_join(v[0], b, is_max);
            }
            warp_reduce_acc<1>(v, is_max ? 1u : 0u);
            if (lane == 0) etot[i] = (double)v[0].s + (double)v[0].c;
        }
        __syncthreads();
        if (ctrl && lane == 0) {
            for (int i = 0; i < 8; ++i) S.row_eval[i] = etot[i];
            S.col_eval_dist[0] = etot[16];
            S.col_eval_dist[1] = etot[17];
            eval_controller(S, etot + 8, blockIdx.x == 0 ? done_count : &ignored);
            const StepScalars sc = step_scalars(S);
            pub = StepPub{sc.cur, 0, S.done, sc.w, sc.tau, (float)(S.eta * S.omega)};
            flag = S.restart_flag;
        }
        __syncthreads();
        if (!ctrl && flag != 0) {  // restart at the current (1) or the average point (2)
            for (int p = warp; p < cp; p += nw) {
                const GridPass t(cpass[p], crows);
                if (t.on && t.sub == 0) {
                    const int j = t.seg;
                    float* c = C + t.local;
                    float* x = pick(V.x0, V.x1, cur) + j;
                    if (flag == 2) {
                        *x = V.x_avg[j];
                        const float kty = c[cur * ncl] = pick(V.kty0, V.kty1, cur)[j] = V.kty_eval[j];
                        float4* rec = records + (size_t)cur * N + j;
                        *rec = make_float4(*x, c[2 * ncl] + kty, rec->z, rec->w);
                    }
                    V.x_last[j] = *x;
                    V.x_acc[j] = make_float2(*x, 0.f);
                    c[3 * ncl] = *x;
                    c[4 * ncl] = 0.f;
                }
            }
            for (int p = warp; p < rp; p += nw) {
                const GridPass t(rpass[p], rrows);
                if (t.on && t.sub == 0) {
                    const int j = t.seg;
                    float* r = R + t.local;
                    float* y = pick(V.y0, V.y1, cur) + j;
                    if (flag == 2) {
                        *y = V.y_avg[j];
                        pick(V.kx0, V.kx1, cur)[j] = r[cur * nrl] = V.kx_eval[j];
                    }
                    V.y_last[j] = *y;
                    V.y_acc[j] = make_float2(*y, 0.f);
                    r[4 * nrl] = *y;
                    r[5 * nrl] = 0.f;
                }
            }
        }
        // (the next step gathers the records that a restart to the average rewrote)
        if (period + 1 < periods && !pub.done && !sync(&ok)) return;
    }
    if (blockIdx.x == 0 && ctrl && lane == 0) {
        *st = S;
        count[32 * kArrive] = sync.turn;  // for the next launch
    }
}

// Plain algorithm (the reference's FP32 PDHG): `checks` times `iterations`
// iterations and the reference's convergence check, on one cluster.  Two
// phases an iteration, no reduction and no controller between checks.  The
// element updates are those of plain_primal_packs / plain_dual_packs; the
// check takes its maxima over the same sums.
__global__ void __launch_bounds__(kResThreads, 1) k_resident_plain(ResArgs A, int iterations, int checks, PlainVecs v,
                                                                   PlainState* st) {
    extern __shared__ char sm[];
    __shared__ PlainState S;  // every block's copy
    __shared__ float wmax[2][32];
    __shared__ float bmax[2][16];
    const int cluster = A.cluster;
    if (st->done) return;  // the whole cluster
    const int rank = cluster > 1 ? (int)cluster_rank() : 0;
    const ResBlock& blk = A.blocks[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int4* rpass = reinterpret_cast<int4*>(sm + A.sm.pass[0]);
    int4* cpass = reinterpret_cast<int4*>(sm + A.sm.pass[1]);
    const char* rrows = sm + A.sm.rows[0];
    const char* crows = sm + A.sm.rows[1];
    float* xs = reinterpret_cast<float*>(sm + A.sm.xs);  // x_bar; x in a check
    float* ys = reinterpret_cast<float*>(sm + A.sm.ys);
    float* C = reinterpret_cast<float*>(sm + A.sm.col);  // x | c | l | u | tau | best x
    float* R = reinterpret_cast<float*>(sm + A.sm.row);  // y | rl | ru | sigma
    const int ncl = A.sm.locals[1], nrl = A.sm.locals[0];
    const int rp = blk.side[0].passes, cp = blk.side[1].passes;
    const int n = A.inst[0].y, m = A.inst[0].w;
    const FromShared gx{xs, n}, gy{ys, m};
    if (threadIdx.x == 0) xs[n] = ys[m] = 0.f;
    load_block<Compact>(A, blk, sm);
    if (threadIdx.x == 0) S = *st;
    for (int k = threadIdx.x; k < m; k += blockDim.x) ys[k] = v.y[k];
    __syncthreads();
    for (int p = warp; p < cp; p += nw) {
        const Pass t(cpass[p], crows);
        if (t.on && t.sub == 0) {
            float* c = C + t.local;
            c[0] = v.x[t.seg];
            c[ncl] = v.c[t.seg];
            c[2 * ncl] = v.l[t.seg];
            c[3 * ncl] = v.u[t.seg];
            c[4 * ncl] = v.tau[t.seg];
            c[5 * ncl] = v.best_x[t.seg];
        }
    }
    for (int p = warp; p < rp; p += nw) {
        const Pass t(rpass[p], rrows);
        if (t.on && t.sub == 0) {
            float* r = R + t.local;
            r[0] = v.y[t.seg];
            r[nrl] = v.rl[t.seg];
            r[2 * nrl] = v.ru[t.seg];
            r[3 * nrl] = v.sigma[t.seg];
        }
    }
    cluster_arrive();  // every block of the cluster runs before the first remote store
    cluster_wait();
    for (int check = 0; check < checks && !S.done; ++check) {
        for (int it = 0; it < iterations; ++it) {
            for (int p = warp; p < cp; p += nw) {
                const Pass t(cpass[p], crows);
                const float aty = pass_dot<false>(t.rows, t.width, t.lg, gy);
                float x_new = 0.f;
                if (t.on) {
                    const float* c = C + t.local;
                    const float x = c[0], l = c[2 * ncl], u = c[3 * ncl];
                    x_new = __fsub_rn(x, __fmul_rn(c[4 * ncl], __fadd_rn(c[ncl], aty)));
                    if (x_new < l) x_new = l;
                    if (x_new > u) x_new = u;
                    push(xs + t.seg, __fsub_rn(__fmul_rn(2.0f, x_new), x), t.sub, 1 << t.lg, cluster);
                }
                __syncwarp();  // every lane of the group has read x
                if (t.on && t.sub == 0) C[t.local] = x_new;
            }
            cluster_arrive();
            cluster_wait();
            for (int p = warp; p < rp; p += nw) {
                const Pass t(rpass[p], rrows);
                const float axbar = pass_dot<false>(t.rows, t.width, t.lg, gx);
                float y = 0.f;
                if (t.on) {
                    const float* r = R + t.local;
                    const float sig = r[3 * nrl];
                    const float w = __fadd_rn(axbar, r[0] / sig);
                    float q = w;
                    if (q < r[nrl]) q = r[nrl];
                    if (q > r[2 * nrl]) q = r[2 * nrl];
                    y = __fmul_rn(sig, __fsub_rn(w, q));
                    push(ys + t.seg, y, t.sub, 1 << t.lg, cluster);
                }
                __syncwarp();
                if (t.on && t.sub == 0) R[t.local] = y;
            }
            cluster_arrive();
            cluster_wait();
        }
        // the check (plain_check_rows / _cols / _finish / _copy_best kernels)
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            if (t.on) push(xs + t.seg, C[t.local], t.sub, 1 << t.lg, cluster);
        }
        cluster_arrive();
        float most[2] = {0.f, 0.f};
        for (int p = warp; p < cp; p += nw) {
            const Pass t(cpass[p], crows);
            const float aty = pass_dot<false>(t.rows, t.width, t.lg, gy);
            if (t.on) {
                const float* c = C + t.local;
                const float x = c[0], tau = c[4 * ncl];
                float proj = __fsub_rn(x, __fmul_rn(tau, __fadd_rn(c[ncl], aty)));
                if (proj < c[2 * ncl]) proj = c[2 * ncl];
                if (proj > c[3 * ncl]) proj = c[3 * ncl];
                most[1] = fmaxf(most[1], fabsf(__fsub_rn(x, proj)) / fmaxf(1e-4f, tau));
            }
        }
        cluster_wait();
        for (int p = warp; p < rp; p += nw) {
            const Pass t(rpass[p], rrows);
            const float ax = pass_dot<false>(t.rows, t.width, t.lg, gx);
            if (t.on) {
                const float rl = R[nrl + t.local], ru = R[2 * nrl + t.local];
                float viol = 0.0f;
                if (rl > -1e15f && ax < rl) viol = fmaxf(viol, __fsub_rn(rl, ax));
                if (ru < 1e15f && ax > ru) viol = fmaxf(viol, __fsub_rn(ax, ru));
                most[0] = fmaxf(most[0], viol);
            }
        }
        for (int h = 0; h < 2; ++h) {
            const float m = warp_max(most[h]);
            if (lane == 0) wmax[h][warp] = m;
        }
        __syncthreads();
        if (warp < 2) {
            const float m = warp_max(lane < nw ? wmax[warp][lane] : 0.f);
            if (lane < cluster) st_rank(map_rank(&bmax[warp][rank], lane), m);
        }
        cluster_arrive();
        cluster_wait();
        if (warp == 0) {
            const float max_p = warp_max(lane < cluster ? bmax[0][lane] : 0.f);
            const float max_d = warp_max(lane < cluster ? bmax[1][lane] : 0.f);
            if (lane == 0) plain_check(S, max_p, max_d);
        }
        __syncthreads();
        if (S.copy_best)
            for (int k = threadIdx.x; k < blk.side[1].locals; k += blockDim.x) C[5 * ncl + k] = C[k];
        __syncthreads();  // the owners move x in the next iteration
    }
    for (int p = warp; p < cp; p += nw) {
        const Pass t(cpass[p], crows);
        if (t.on && t.sub == 0) {
            v.x[t.seg] = C[t.local];
            v.best_x[t.seg] = C[5 * ncl + t.local];
        }
    }
    for (int p = warp; p < rp; p += nw) {
        const Pass t(rpass[p], rrows);
        if (t.on && t.sub == 0) v.y[t.seg] = R[t.local];
    }
    if (rank == 0 && threadIdx.x == 0) *st = S;
}

namespace {

// Entries of every pass from the (renumbered, scaled) matrix: a warp per pass.
// place: {first pair, width, first segment in the batch, segments}, then
// {the other side's first index, side, lanes, the other side's length}.
template <class Entries>
__global__ void k_resident_fill(int npass, const int4* __restrict__ place, SegMatrix R, SegMatrix C,
                                char* __restrict__ rows) {
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); p < npass; p += nw) {
        const int4 t = place[2 * p];
        const int4 o = place[2 * p + 1];
        const SegMatrix& A = o.y ? C : R;
        const int L = o.z, sub = lane & (L - 1), g = lane / L;
        const int none = Entries::kPair == Compact::kPair ? o.w : -1;
        int k = 0, e = 0;
        if (g < t.w) {
            k = A.ptr[t.z + g] + sub;
            e = A.ptr[t.z + g + 1];
        }
        char* out = rows + (size_t)t.x * Entries::kPair;
        for (int r = 0; r < t.y; r += 2, k += 2 * L, out += Entries::kPair) {
            const int2 v = k < e ? A.pairs[k] : make_int2(none + o.x, 0);
            const int2 w = k + L < e ? A.pairs[k + L] : make_int2(none + o.x, 0);
            Entries::store(out, v.x - o.x, __int_as_float(v.y), w.x - o.x, __int_as_float(w.y));
        }
    }
}

}  // namespace

void ResidentPlan::release() {
    ready_ = false;
    tab_.release();
    rows_.release();
    slots_.release();
    esums_.release();
}

int ResidentPlan::build(const std::vector<int>& csr_ptr, const std::vector<int>& csc_ptr, const std::vector<int>& roff,
                        const std::vector<int>& coff, const std::vector<uint8_t>& row_lanes,
                        const std::vector<uint8_t>& col_lanes, int sm_count, cudaStream_t s, Kind kind, double most_us) {
    release();
    kind_ = kind;
    const bool plain = kind == kPlain, grid = kind == kGrid;
    const void* kernel = plain  ? (const void*)k_resident_plain
                         : grid ? (const void*)k_resident_grid
                                : (const void*)k_resident_steps;
    const long long pair_bytes = grid ? Wide::kPair : Compact::kPair;
    const int col_words = plain ? kPlainColWords : grid ? kGridColWords : kColWords;
    const int row_words = plain ? kPlainRowWords : grid ? kGridRowWords : kRowWords;
    const int B = (int)roff.size() - 1;
    instances_ = B;
    int dev = 0, optin = 0;
    SIHG_CUDA(cudaGetDevice(&dev));
    SIHG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa{};
    SIHG_CUDA(cudaFuncGetAttributes(&fa, kernel));
    const int budget = optin - (int)fa.sharedSizeBytes;
    const std::vector<int>* ptrs[2] = {&csr_ptr, &csc_ptr};
    const std::vector<int>* offs[2] = {&roff, &coff};
    const std::vector<uint8_t>* lanes[2] = {&row_lanes, &col_lanes};
    // the smallest instance bound: both copies and both sides of the matrix
    // over 16 blocks must fit; most batches end here
    for (int b = 0; b < B; ++b) {
        const double nnz = csr_ptr[roff[b + 1]] - csr_ptr[roff[b]], m = roff[b + 1] - roff[b], n = coff[b + 1] - coff[b];
        if (!grid && (m > 0xfffe || n > 0xfffe)) return SIH_PDHG_OK;  // 16-bit indices
        if (grid) {
            if ((16.0 * nnz + 4.0 * (col_words * n + row_words * m)) / sm_count > budget) return SIH_PDHG_OK;
        } else if (4.0 * (m + n) + (12.0 * nnz + 4.0 * (col_words * n + row_words * m)) / 16.0 > budget) return SIH_PDHG_OK;
    }
    // every instance's passes: {first segment, segments, width, log2 L}, rows of A then columns
    std::vector<int4> inst(B), all;
    std::vector<size_t> first(2 * (size_t)B + 1, 0);
    for (int b = 0; b < B; ++b) {
        inst[b] = make_int4(coff[b], coff[b + 1] - coff[b], roff[b], roff[b + 1] - roff[b]);
        for (int h = 0; h < 2; ++h) {
            const std::vector<int>& ptr = *ptrs[h];
            const uint8_t* ln = lanes[h]->data();
            const int s1 = (*offs[h])[b + 1];
            for (int seg = (*offs[h])[b]; seg < s1;) {
                const int L = ln[seg];
                int e = seg, width = 0, lg = 0;
                while ((1 << lg) < L) ++lg;
                while (e < s1 && e - seg < 32 / L && ln[e] == L) {
                    width = std::max(width, (ptr[e + 1] - ptr[e] + L - 1) / L);
                    ++e;
                }
                all.push_back(make_int4(seg, e - seg, width, lg));
                seg = e;
            }
            first[2 * b + h + 1] = all.size();
        }
    }
    // calls f(pass, block of C) for the passes of an instance's side
    auto deal = [&](int b, int h, int C, auto&& f) {
        const size_t a0 = first[2 * b + h], a1 = first[2 * b + h + 1];
        for (size_t q0 = a0; q0 < a1;) {
            size_t q1 = q0;  // runs of equal lanes and width
            while (q1 < a1 && all[q1].z == all[q0].z && all[q1].w == all[q0].w) ++q1;
            const long long len = (long long)(q1 - q0);
            for (size_t q = q0; q < q1; ++q) {
                int r;
                if (grid) {
                    // each run spread evenly in its order: segments of one length keep the caller's
                    // order, so that a block gets the same part of the LP from every run and side,
                    // and its gathers, where the LP has a block structure, meet in its L1
                    r = (int)((long long)(q - q0) * C / len);
                    if (len < C) r = (int)((r + C / (2 * len)) % C);
                } else {  // the passes run by descending length: dealt out back and forth
                    const int t = (int)((q - a0) % (2 * (size_t)C));
                    r = t < C ? t : 2 * C - 1 - t;
                }
                f(all[q], r);
            }
            q0 = q1;
        }
    };
    ResSmem sm{};
    int sides[2] = {0, 0};  // most passes of a block, by side
    auto measure = [&](int C) -> int {  // the shared memory layout for clusters of C; most passes of a block
        long long mrows[2] = {0, 0};
        int mpass[2] = {0, 0}, mloc[2] = {0, 0}, mn = 0, mm = 0;
        std::vector<int> npass(C), nloc(C);
        std::vector<long long> nrow(C);
        for (int b = 0; b < B; ++b) {
            mn = std::max(mn, inst[b].y);
            mm = std::max(mm, inst[b].w);
            for (int h = 0; h < 2; ++h) {
                std::fill(npass.begin(), npass.end(), 0);
                std::fill(nloc.begin(), nloc.end(), 0);
                std::fill(nrow.begin(), nrow.end(), 0);
                deal(b, h, C, [&](const int4& p, int r) {
                    npass[r] += 1;
                    nloc[r] += p.y;
                    nrow[r] += (p.z + 1) / 2;
                });
                mpass[h] = std::max(mpass[h], *std::max_element(npass.begin(), npass.end()));
                mloc[h] = std::max(mloc[h], *std::max_element(nloc.begin(), nloc.end()));
                mrows[h] = std::max(mrows[h], *std::max_element(nrow.begin(), nrow.end()));
            }
        }
        long long at = 0;
        auto put = [&](long long bytes) {
            const long long a = at;
            at = (at + bytes + 15) & ~15ll;
            return (int)std::min<long long>(a, INT32_MAX);
        };
        for (int h = 0; h < 2; ++h) sm.rows[h] = put(pair_bytes * mrows[h]);
        for (int h = 0; h < 2; ++h) sm.pass[h] = put(16ll * mpass[h]);
        sm.xs = put(grid ? 0 : 4ll * (mn + 1));
        sm.ys = put(grid ? 0 : 4ll * (mm + 1));
        sm.locals[0] = mloc[0];
        sm.locals[1] = mloc[1];
        sm.col = put(4ll * col_words * mloc[1]);
        sm.row = put(4ll * row_words * mloc[0]);
        const int warps = grid ? 32 : kResWarps;
        sm.seg = put(kind == kCluster ? 2ll * mloc[1] : 0);
        sm.red = put((long long)sizeof(Sums) * (warps + 16));
        sm.eval = put(plain ? 0 : kEvalQ * (8ll * warps + 8ll * 16 + 8));
        sm.total = (int)std::min<long long>(at, INT32_MAX);
        sides[0] = mpass[0];
        sides[1] = mpass[1];
        return std::max(mpass[0], mpass[1]);
    };
    // The smallest cluster that holds an instance; a larger one while SMs are
    // left over and a block has more than 8 passes a side (two warps per
    // scheduler): beyond that the barriers and pushes of more blocks cost what
    // the shorter phases save (317 x 803: 4 blocks of 9 passes and 8 of 5 are
    // equal).
    int C = grid ? sm_count : 1, most = measure(C);
    while (!grid && C < 16 && sm.total > budget) most = measure(C *= 2);
    if (sm.total > budget) return SIH_PDHG_OK;
    while (!grid && C < 16 && (long long)B * 2 * C <= sm_count && most > 8) most = measure(C *= 2);
    // as few warps as do both sides in the same rounds (grid form: a thread per block sums)
    int nw = grid ? kGridThreads / 32 - 1 : std::max(1, std::min(kResThreads / 32 - 1, most));
    auto rounds = [&](int w) { return (sides[0] + w - 1) / w + (sides[1] + w - 1) / w; };
    while (!grid && nw > 1 && rounds(nw - 1) == rounds(nw)) --nw;
    threads_ = 32 * (nw + 1);
    if (grid && sm_count > threads_) return SIH_PDHG_OK;
    npass_ = (int)all.size();
    SIHG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, budget));
    if (grid) {
        int occ = 0, coop = 0;
        SIHG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        SIHG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads_, sm.total));
        if (!coop || occ < 1) return SIH_PDHG_OK;
        SIHG_TRY(slots_.alloc(sizeof(unsigned) * 32 * (kArrive + 1) + sizeof(Sums) * (size_t)C));
        SIHG_TRY(esums_.alloc(sizeof(float2) * kEvalQ * (size_t)C));
    } else {
        SIHG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    int clusters = sm_count;  // at a time; blocks that share an SM gain nothing over taking turns
    if (!grid && C > 1) {
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {(unsigned)C, 1, 1};
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(B * C));
        cfg.blockDim = dim3((unsigned)threads_);
        cfg.dynamicSmemBytes = (size_t)sm.total;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            return SIH_PDHG_OK;
        }
    }
    if (kind == kCluster && B > clusters && most_us > 0.0) {
        // Every instance takes the cluster that the largest one needs, and the
        // clusters take turns (many of them overlap).  A turn's step takes 4.7 us for its
        // barriers and controller alone, up to 9.3 us where an instance fills its
        // cluster's memory.  Estimated / measured us per step: 64 of 2,000 x 5,000 (clusters
        // of 4) 18.5 / 18.6, 512 of 1,000 x 2,500 (2) 62 / 63, 48 of 5,000 x 12,000 (16) 62 /
        // 64, 64 of 200 to 3,000 rows (8) 32 / 30, 200 of 100 to 3,000 (8) 100 / 90, 300 of
        // 200 x 500 with one of 5,000 x 12,000 (16) 215 / 207.
        double sum = 0.0;
        for (int b = 0; b < B; ++b) {
            double bytes = 4.0 * (col_words + C) * inst[b].y + 4.0 * (row_words + C) * inst[b].w;
            for (size_t q = first[2 * (size_t)b]; q < first[2 * (size_t)b + 2]; ++q) bytes += pair_bytes * ((all[q].z + 1) / 2);
            const double full = std::min(1.0, bytes / ((double)C * budget));
            sum += 4.7 + 4.6 * full * (2.0 - full);
        }
        double turns = (double)B / clusters;
        if (turns < 4.0) turns = std::ceil(turns);
        if (turns * sum / B > most_us) return SIH_PDHG_OK;
    }
    // the tables: blocks, instances, passes by block, and each pass's place in the matrix for the fill
    const size_t nb = sizeof(ResBlock) * (size_t)B * C, ni = sizeof(int4) * (size_t)B, np = sizeof(int4) * all.size();
    const size_t o_i = (nb + 15) & ~(size_t)15, o_p = o_i + ni, o_l = o_p + np;
    std::vector<char> buf(o_l + 2 * np);
    ResBlock* blocks = reinterpret_cast<ResBlock*>(buf.data());
    std::memcpy(buf.data() + o_i, inst.data(), ni);
    int4* passes = reinterpret_cast<int4*>(buf.data() + o_p);
    int4* place = reinterpret_cast<int4*>(buf.data() + o_l);
    long long rows = 0;
    {
        std::vector<int> next(C);
        int at = 0;
        for (int b = 0; b < B; ++b)
            for (int h = 0; h < 2; ++h) {
                ResBlock* blk = blocks + (size_t)b * C;
                for (int r = 0; r < C; ++r) blk[r].side[h] = ResSide{};
                deal(b, h, C, [&](const int4& p, int r) {
                    blk[r].side[h].passes += 1;
                    blk[r].side[h].rows += (p.z + 1) / 2;
                });
                for (int r = 0; r < C; ++r) {
                    ResSide& sd = blk[r].side[h];
                    next[r] = sd.pass_begin = at;
                    at += sd.passes;
                    sd.row_begin = (int)rows;
                    rows += sd.rows;
                    sd.rows = 0;  // counted again below
                }
                deal(b, h, C, [&](const int4& p, int r) {
                    ResSide& sd = blk[r].side[h];
                    const int k = next[r]++;
                    passes[k] = make_int4(sd.rows, p.z | (p.w << 24), p.x - (*offs[h])[b], sd.locals | (p.y << 24));
                    place[2 * (size_t)k] = make_int4(sd.row_begin + sd.rows, p.z, p.x, p.y);
                    place[2 * (size_t)k + 1] = make_int4((*offs[1 - h])[b], h, 1 << p.w, (*offs[1 - h])[b + 1] - (*offs[1 - h])[b]);
                    sd.rows += (p.z + 1) / 2;
                    sd.locals += p.y;
                });
            }
    }
    SIHG_TRY(tab_.alloc(buf.size()));
    SIHG_CUDA(cudaMemcpyAsync(tab_.as<void>(), buf.data(), buf.size(), cudaMemcpyHostToDevice, s));
    SIHG_TRY(rows_.alloc((size_t)pair_bytes * (size_t)std::max<long long>(1, rows)));
    char* d = tab_.as<char>();
    args_ = ResArgs{(const ResBlock*)d, (const int4*)(d + o_i), (const int4*)(d + o_p), rows_.as<char>(), sm, C};
    ready_ = true;
    return SIH_PDHG_OK;
}

int ResidentPlan::fill(const SegMatrix& rows_A, const SegMatrix& cols_A, cudaStream_t s) {
    const int4* place = args_.passes + npass_;
    const int g = std::max(1, std::min(1216, (npass_ + 7) / 8));
    if (kind_ == kGrid)
        k_resident_fill<Wide><<<g, 256, 0, s>>>(npass_, place, rows_A, cols_A, rows_.as<char>());
    else
        k_resident_fill<Compact><<<g, 256, 0, s>>>(npass_, place, rows_A, cols_A, rows_.as<char>());
    SIHG_LAUNCH_CHECK();
    return SIH_PDHG_OK;
}

// The launch configuration of one cluster per instance.
cudaLaunchConfig_t ResidentPlan::config(cudaLaunchAttribute* at, cudaStream_t s) const {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)args_.cluster, 1, 1};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(instances_ * args_.cluster));
    cfg.blockDim = dim3((unsigned)threads_);
    cfg.dynamicSmemBytes = (size_t)args_.sm.total;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

int ResidentPlan::launch(int nsteps, int periods, const Vecs& V, Inst* st, unsigned* done_count,
                         cudaStream_t s) const {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(at, s);
    SIHG_CUDA(cudaLaunchKernelEx(&cfg, k_resident_steps, args_, nsteps, periods, V, st, done_count));
    return SIH_PDHG_OK;
}

int ResidentPlan::reset(cudaStream_t s) {
    if (kind_ == kGrid) SIHG_CUDA(cudaMemsetAsync(slots_.as<void>(), 0, slots_.bytes(), s));
    return SIH_PDHG_OK;
}

int ResidentPlan::launch_grid(int nsteps, int periods, const Vecs& V, Inst* st, unsigned* done_count, float4* records,
                              int N, const GridBar& gb, cudaStream_t s) const {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = config(at, s);
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_resident_grid, args_, nsteps, periods, V, st, done_count, records,
                                             N, slots_.as<unsigned>(), reinterpret_cast<Sums*>(slots_.as<unsigned>() + 32 * (kArrive + 1)), esums_.as<float2>(), gb);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // the device cannot hold the whole grid now; the caller falls back
        (void)cudaGetLastError();
        return SIH_PDHG_ERR_UNSUPPORTED;
    }
    if (e != cudaSuccess) return cuda_fail(e, "resident grid kernel launch", __FILE__, __LINE__);
    return SIH_PDHG_OK;
}

int ResidentPlan::launch_plain(int iterations, int checks, const PlainVecs& v, PlainState* st, cudaStream_t s) const {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(at, s);
    SIHG_CUDA(cudaLaunchKernelEx(&cfg, k_resident_plain, args_, iterations, checks, v, st));
    return SIH_PDHG_OK;
}

}  // namespace sihg
