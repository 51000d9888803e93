// A block of activity steps of a network WITH synapses in one launch: the
// parts shared by the FP64 (activity.cu) and FP32 (fp32.cu) kernels.
//
// A step's input needs every spike of the step before, so the thread blocks
// meet at a barrier between steps.  One launch per step pays that as a launch
// (launch, constant loads, state loads and drain, also when the network fills a
// fraction of the device); here all thread blocks are resident together, the
// state stays in registers, and the barrier is split: a block arrives when its
// spikes are pushed and then does what does not depend on the others
// (calcium, growth, the draws of the coming steps) before it waits.  Bound by
// the chain of a step: pushed sum past L1, ten dependent substeps, the spikes'
// edges, the barrier.  Microseconds per step, one launch per step -> here:
// FP64 2,000 neurons 6.6 -> 3.3, 51,842 8.3 -> 3.8, 113,000 9.3 -> 4.9; FP32
// 5.0 -> 2.5, 6.3 -> 3.3, 6.6 -> 3.6; AEIF FP64 100,003 12.0 -> 7.4.
//
// Up to kCoupledCluster thread blocks form one cluster and use the hardware's
// cluster barrier (6,100 neurons: 3.4 us per step FP64, 2.6 FP32); more are
// launched cooperatively (the launch fails rather than leave one of them out)
// and count arrivals in device memory (6,200 neurons: 3.7 and 3.1 us).
// More neurons than resident threads run in rounds, several per thread with
// their state in shared memory (up to 1,136,640 neurons FP64, 1,875,456 FP32;
// one launch per step -> here, four synapses per neuron: FP64 300,000 neurons
// 14.4 -> 11.8, 600,000 24.9 -> 21.2, 1M 38.6 -> 32.0 (37.9 with the shape the
// tuner picks); FP32 9.4 -> 6.3, 14.4 -> 10.0, 21.4 -> 14.3 (tuned 19.6)).
#pragma once

#include <algorithm>

#include "rl_context.cuh"

namespace rl {

constexpr int kCoupledBlock = 384;          // threads (neurons) per block, two blocks per SM
constexpr unsigned kCoupledCluster = 16;    // blocks per cluster (8 are portable)
constexpr uint32_t kCoupledChunk = 16;      // steps between two replays of calcium and growth (bits of a uint16_t)

// The barrier between the steps of a launch that counts arrivals.
struct StepBarrier {
    uint32_t* count;  // arrivals, in device memory
    uint32_t* lost;   // the context's word in pinned host memory, set when a wait gives up
    uint32_t polls;   // after so many polls
};

#if defined(__CUDACC__)
// This block's pushes of the step are issued by all its threads.
template <bool CLUSTER>
__device__ __forceinline__ void step_arrive(const StepBarrier& bar) {
    if constexpr (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    } else {
        __syncthreads();
        if (threadIdx.x == 0) {
            // a release at device scope, which covers what the block's other
            // threads wrote before the barrier above
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar.count) : "memory");
        }
    }
}

// Waits until `arrivals` arrivals are counted; false (in every thread of the
// block) if the bounded wait ran out, which the host reads in *bar.lost: the
// blocks that gave up have not written their state, so it is no state any more.
template <bool CLUSTER>
__device__ __forceinline__ bool step_wait(const StepBarrier& bar, uint32_t arrivals) {
    if constexpr (CLUSTER) {
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        return true;
    } else {
        int late = 0;
        if (threadIdx.x == 0) {
            uint32_t polls = 0, seen = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar.count) : "memory");
            } while ((int32_t)(seen - arrivals) < 0 && ++polls < bar.polls);
            if ((int32_t)(seen - arrivals) < 0) {
                *(volatile uint32_t*)bar.lost = 1u;
                late = 1;
            }
        }
        return __syncthreads_or(late) == 0;
    }
}

// Neuron i's sum pushed at the step before, read past L1 (other SMs' atomics
// wrote it) and cleared.
template <typename T>
__device__ __forceinline__ T take_pushed(T* in, uint32_t i) {
    const T s = __ldcg(in + i);
    if (s != 0) {
        __stcg(in + i, (T)0);
    }
    return s;
}

__device__ __forceinline__ void add_weight(long long* p, int32_t w) {
    atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)(long long)w);  // two's complement: the signed sum
}
__device__ __forceinline__ void add_weight(int32_t* p, int32_t w) {
    atomicAdd(p, w);
}

// The warp's spikes: each firing lane's out-edges o0 .. o1 go to their
// targets' sums of the next step, four spikes at a time with eight lanes each,
// so that the edges' dependent loads lie side by side.
template <typename T>
__device__ __forceinline__ void push_warp(bool f, uint32_t o0, uint32_t o1, const uint32_t* __restrict__ out_perm, const uint32_t* __restrict__ tgt,
                                          const int32_t* __restrict__ w, T* next) {
    uint32_t m = __ballot_sync(0xFFFFFFFFu, f);
    const uint32_t g = (threadIdx.x & 31u) >> 3, sub = threadIdx.x & 7u;
    while (m) {
        const uint32_t m1 = m & (m - 1u), m2 = m1 & (m1 - 1u), m3 = m2 & (m2 - 1u);
        const uint32_t mine = g == 0u ? m : (g == 1u ? m1 : (g == 2u ? m2 : m3));  // its lowest lane is the group's spike
        const int s = mine ? __ffs((int)mine) - 1 : 0;
        const uint32_t b0 = __shfl_sync(0xFFFFFFFFu, o0, s), b1 = __shfl_sync(0xFFFFFFFFu, o1, s);
        if (mine) {
            for (uint32_t j = b0 + sub; j < b1; j += 8u) {
                const uint32_t e = out_perm[j];
                add_weight(next + tgt[e], w[e]);
            }
        }
        m = m3 & (m3 - 1u);
    }
    __syncwarp();
}

// Edges j, j + 8, ... below end of the out-CSR order, four at a time, so that
// their dependent loads lie side by side (one at a time -> four, us per step:
// 600,000 neurons with 20 synapses each FP64 29.4 -> 25.1, FP32 18.8 -> 14.2;
// 300,000 with 100 71.4 -> 68.8 and 67.9 -> 61.0).
template <typename T>
__device__ __forceinline__ void push_edges(uint32_t j, uint32_t end, const uint32_t* __restrict__ out_perm, const uint32_t* __restrict__ tgt,
                                           const int32_t* __restrict__ w, T* next) {
    for (; j < end; j += 32u) {
        uint32_t e[4], t[4];
        int32_t v[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            e[q] = j + 8u * q < end ? out_perm[j + 8u * q] : 0u;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            t[q] = j + 8u * q < end ? tgt[e[q]] : 0u;
            v[q] = j + 8u * q < end ? w[e[q]] : 0;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            if (j + 8u * q < end) {
                add_weight(next + t[q], v[q]);
            }
        }
    }
}

// The block's queued spikes (neurons base + who[q]), eight lanes each.
template <int BLOCK, typename T>
__device__ __forceinline__ void push_queue(uint32_t cnt, uint32_t base, const uint16_t* who, const uint32_t* __restrict__ out_off,
                                           const uint32_t* __restrict__ out_perm, const uint32_t* __restrict__ tgt, const int32_t* __restrict__ w,
                                           T* next) {
    for (uint32_t q = threadIdx.x >> 3; q < cnt; q += BLOCK / 8) {
        const uint32_t i = base + who[q];
        push_edges(out_off[i] + (threadIdx.x & 7u), out_off[i + 1], out_perm, tgt, w, next);
    }
}

// Appends `slot` of the lanes with `take` set to the queue.  All lanes call it.
__device__ __forceinline__ void queue_slots(bool take, uint32_t slot, uint16_t* who, uint32_t* cnt) {
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, take);
    if (mask == 0u) {
        return;
    }
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t first = 0;
    if (lane == 0) {
        first = atomicAdd(cnt, (uint32_t)__popc(mask));
    }
    first = __shfl_sync(0xFFFFFFFFu, first, 0);
    if (take) {
        who[first + (uint32_t)__popc(mask & ((1u << lane) - 1u))] = (uint16_t)slot;
    }
}
#endif

// The polls of a wait: one neuron may hold every synapse, and its block then
// walks the list alone while the others wait (up to 75 ns per synapse; a poll
// takes about 700).
inline uint32_t barrier_polls(const Ctx& c) {
    return (uint32_t)std::min<uint64_t>(0xFFFFFFFFull, c.wait_polls + c.graph.num_edges / 2u);
}

inline StepBarrier step_barrier(const Ctx& c) {
    return StepBarrier{ c.act_bar.p, c.lost_word(), barrier_polls(c) };
}

// Launches the coupled kernel of `steps` steps (its cluster form for few blocks) if all its
// thread blocks can be resident together; false if not.
template <typename... KArgs, typename... Args>
bool launch_coupled(Ctx& c, uint32_t steps, void (*cluster_kernel)(KArgs...), void (*grid_kernel)(KArgs...), Args... args) {
    const unsigned blocks = blocks_for(c.n, kCoupledBlock);
    const bool cluster = blocks <= kCoupledCluster;
    void (*kernel)(KArgs...) = cluster ? cluster_kernel : grid_kernel;
    if (cluster) {
        RL_CUDA_TRY(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    } else {
        int per_sm = 0;
        RL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, kCoupledBlock, 0));
        if (blocks > (unsigned)per_sm * (unsigned)c.num_sms) {
            return false;
        }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kCoupledBlock);
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = blocks;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PhaseScope ps(c, PH_ACTIVITY_KERNEL, steps);
    if (cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...) != cudaSuccess) {
        (void)cudaGetLastError();  // such a launch is not available here: the caller takes one launch per step
        return false;
    }
    if (g_bind.launches) {
        ++*g_bind.launches;
    }
    return true;
}

// Whether a block of `steps` steps in `rounds` neurons for each of `threads`
// threads beats one launch per step (us per step, one launch per step against
// rounds).  It does for the Izhikevich and Poisson models (above) unless
//   * the synapse list is so long that walking it at each step's end, with
//     nothing beside it, takes longer than the rest: FP64 30M synapses 74, 63
//     (1M neurons) and 67.8, 68.8 (300,000), 36M 67.8, 68.9, 40M 85, 91, 60M
//     121, 188; FP32 40M 71.6, 45.4, 50M 88.9, 80.8, 60M 102, 104 and 116, 150;
//   * FP64 has only two steps to spread its loads and stores over: 850,000
//     neurons 41.1, 43.0 (three steps 46.1, 38.5).
// The other models' longer substeps leave less to gain: AEIF FP64 400,000
// neurons (4 rounds) 26.6, 25.5, 700,000 (7) 42.4, 44.5; FitzHugh-Nagumo, of
// whose neurons two in five fire at a step, FP64 300,000 (3) 20.1, 19.4,
// 400,000 (4) 23.6, 24.9; FP32 where the last round is nearly full: 500,000 (3
// rounds, 98 %) 20.7, 18.8, 700,000 (5, 82 %) 26.8, 29.0, 250,000 (2, 73 %)
// 13.9, 13.1, 200,000 (2, 59 %) 9.8, 10.9, and the L1 cache is left some room:
// 1.4M (9) 60.5, 59.4, 1.87M (11) 92.6, 129.
inline bool rounds_pay(const Ctx& c, uint32_t steps, uint32_t rounds, uint64_t threads) {
    const bool fp32 = is_fp32(c);
    if (c.graph.num_edges > (fp32 ? 56'000'000u : 32'000'000u) || (!fp32 && steps < 3)) {
        return false;
    }
    if (c.cfg.neuron_model == RL_MODEL_AEIF) {
        return fp32 || rounds <= 4;
    }
    if (c.cfg.neuron_model == RL_MODEL_FITZHUGH_NAGUMO) {
        const double used = (double)c.n / (double)(rounds * threads);
        return fp32 ? rounds <= 9 && used >= (rounds == 2 ? 0.7 : 0.9) : rounds <= 3;
    }
    return true;
}

// The form for more neurons than resident threads: `rounds` neurons per
// thread, their x, u and draws in shared memory (`bytes` per neuron), at most
// `per_sm_target` blocks per SM; false where they do not all fit, or would not
// be faster.  `bar` is the barrier as the kernel takes it.
template <typename Args, typename... Bar>
bool launch_coupled_rounds(Ctx& c, uint32_t steps, void (*kernel)(Args, const ActDesc*, uint32_t, uint32_t, uint8_t*, Bar...), unsigned per_sm_target,
                           size_t bytes, const Args& args, uint8_t* fired_before_last, Bar... bar) {
    const unsigned slots = per_sm_target * (unsigned)c.num_sms;
    const uint32_t rounds = blocks_for(c.n, slots * kCoupledBlock);
    const unsigned blocks = blocks_for(c.n, rounds * kCoupledBlock);
    const size_t smem = bytes * rounds * kCoupledBlock;
    constexpr size_t kFixed = 1024;  // at least the kernels' static shared memory
    if (!rounds_pay(c, steps, rounds, (uint64_t)slots * kCoupledBlock) || rounds * kCoupledBlock > 65536u || smem > (size_t)c.smem_optin - kFixed) {
        return false;
    }
    allow_shared_memory(c, kernel, kFixed);
    int per_sm = 0;
    RL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, kCoupledBlock, smem));
    if (blocks > (unsigned)per_sm * (unsigned)c.num_sms) {
        return false;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kCoupledBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PhaseScope ps(c, PH_ACTIVITY_KERNEL, steps);
    if (cudaLaunchKernelEx(&cfg, kernel, args, (const ActDesc*)c.act_desc.p, steps, rounds, fired_before_last, bar...) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    if (g_bind.launches) {
        ++*g_bind.launches;
    }
    return true;
}

}  // namespace rl
