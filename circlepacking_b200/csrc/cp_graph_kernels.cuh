// Kernels of the graph engine: the depth-first refinement kernel, and the
// persistent level kernel with the proposal network inline.  Instantiated per
// precision in cp_graph_fp64.cu / cp_graph_fp32.cu so the two compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include "cp_level.cuh"
#include "cp_refine.cuh"
#include "cp_tc.cuh"

namespace cpb {

// Block-size variants of the depth-first kernel (the values of
// cp_refine_opts.block) with the threads and the register cap of each.
constexpr int kGraphVariants = 5;
constexpr int kGraphBlock[kGraphVariants] = {64, 128, 256, 512, 1024};
__host__ __device__ constexpr int deep_regs(int block) { return block >= 1024 ? 80 : block >= 512 ? 96 : 128; }
__host__ __device__ constexpr int deep_threads(int block) { return block >= 1024 ? 384 : block >= 512 ? 320 : block; }

template <int FAM, int BLOCK>
struct DeepSmem {
    LevelCounts counts;
    WarpBoxes<family_dims(FAM)> warp[deep_threads(BLOCK) / 32];
};

// One round of a depth-first refinement (cp_refine.cuh).  The last block to finish
// prepares the next round, if any parcel is left over.
template <int FAM, int PREC, int BLOCK>
__global__ void __launch_bounds__(deep_threads(BLOCK)) __maxnreg__(deep_regs(BLOCK))
    k_refine_deep(RefineArgs r) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<DeepSmem<FAM, BLOCK>*>(smem_raw);
    constexpr unsigned kWarps = deep_threads(BLOCK) / 32;
    level_smem_init(sm.counts);
    __syncthreads();
    unsigned handles = 0;
    const unsigned w = threadIdx.x >> 5;
    refine_warp<FAM, PREC, true>(r, sm.counts, sm.warp[w], gridDim.x * kWarps, blockIdx.x * kWarps + w, handles);
    level_flush(r.level, sm.counts, handles);
    __threadfence();
    __syncthreads();
    if (threadIdx.x != 0) return;
    DeepSched& s = *r.sched;
    if (atomicAdd(&s.done, 1u) + 1u != gridDim.x) return;
    __threadfence();
    const unsigned left = *(volatile unsigned*)&s.filled - *(volatile unsigned*)&s.taken;
    const unsigned parcels = *(volatile unsigned*)&s.parcels;
    s.rounds += 1;
    s.left = left;
    s.epoch += 1;
    s.inputs = parcels < r.slots ? parcels : r.slots;
    s.given += *(volatile unsigned*)&s.filled;
    s.ticket = gridDim.x * kWarps;
    s.parcels = s.filled = s.taken = s.idle = s.done = 0;
}

struct PersistArgs {
    const BoxList* levels;  // device array [nlevels]
    DevSched* sched;
    unsigned long long* cnt;
    unsigned long long* per_depth;
    SingleTable tab;
    int policy, max_depth;
    double lambda_scale;
    int digest;
};

// The persistent level kernel with the proposal network run inline: a CTA of
// 128 threads claims 128 boxes of the job at a time, computes their features,
// runs the network's forward pass on the tensor cores (tcgen05, accumulators in
// 64 tensor-memory columns, tc::net_forward), and each thread evaluates its box
// with the criterion order and split axis the network proposes.  The verdicts
// are the interval kernels' own; a timed-out tensor-core wait raises E_TC.
struct NetArgs {
    const tc::bf16* views;
    const float* master;
    int wait_limit;
    int want_order, want_axis;
};
constexpr int kNetBlock = tc::kTcRows;  // one box per thread of a 128-thread CTA
constexpr int kNetMaxCtasPerSm = 512 / (int)tc::kNetCols;  // tensor memory: 512 columns per SM

// (__launch_bounds__ with 5 resident CTAs caps the registers near 96)
template <int FAM, int PREC>
__global__ void __launch_bounds__(kNetBlock, 5) k_level_persist_net(PersistArgs pa, NetArgs na) {
    constexpr int D = family_dims(FAM);
    __shared__ LevelSmem<kNetBlock / 32> sm;
    __shared__ __align__(128) tc::NetSmem net;
    __shared__ unsigned long long claim;
    const DevJob job = pa.sched->job;
    if (job.count == 0) return;  // uniform over the grid
    LevelArgs a;
    a.in = pa.levels[job.in_level];
    a.begin = job.begin;
    a.count = job.count;
    a.out = job.out_level >= 0 ? pa.levels[job.out_level] : BoxList{nullptr, nullptr, nullptr, 0};
    a.cnt = pa.cnt;
    a.per_depth = pa.per_depth;
    a.tab = pa.tab;
    a.policy = pa.policy;
    a.lambda_scale = pa.lambda_scale;
    a.max_depth = job.out_level >= 0 ? pa.max_depth : 0;
    a.axis_hint = nullptr;
    a.order_hint = nullptr;
    a.digest = pa.digest;
    level_smem_init(sm);
    tc::net_setup(net, na.views, na.master);
    __syncthreads();
    unsigned handles = 0;
    bool ok = true;
    for (;;) {
        if (threadIdx.x == 0) claim = atomicAdd(&pa.sched->claim, (unsigned long long)kNetBlock);
        __syncthreads();
        const unsigned long long start = claim;
        __syncthreads();  // every thread has read the claim before it is replaced
        if (start >= job.count) break;  // uniform over the CTA
        const size_t j = (size_t)(start + threadIdx.x);
        float f[tc::NK];
        if (j < job.count) {
            const size_t i = a.begin + j;
            double lo[4], hi[4];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                lo[d] = a.in.lo[d * a.in.cap + i];
                hi[d] = a.in.hi[d * a.in.cap + i];
            }
            const int dep = a.in.depth[i];
            tc::box_features_fast<D>(lo, hi, dep == 0xFF ? 0 : dep, f);
        } else {
#pragma unroll
            for (int k = 0; k < tc::NK; ++k) f[k] = 0.f;
        }
        float z[tc::NO];
        if (!(ok = tc::net_forward(net, f, z, na.wait_limit))) break;
        int ord = -1, ax = -1;
        if (na.want_order) {
            if (FAM == F_MIDDLE)
                ord = fmaxf(z[2], z[3]) > fmaxf(z[0], z[1]) ? 1 : 0;
            else if (FAM == F_END_2D || FAM == F_END_3D)
                ord = z[1] > z[0] ? 1 : 0;
            else
                ord = 0;
        }
        if (na.want_axis) {
            ax = 0;
            float best = z[4];
#pragma unroll
            for (int d = 1; d < D; ++d)
                if (z[4 + d] > best) {
                    best = z[4 + d];
                    ax = d;
                }
        }
        level_step<FAM, PREC>(a, j, sm, handles, ord, ax);
    }
    if (!ok && threadIdx.x == 0) atomicOr(&a.cnt[C_ERR], (unsigned long long)E_TC);
    tc::net_teardown(net, ok);
    level_flush(a, sm, handles);
}

}  // namespace cpb
