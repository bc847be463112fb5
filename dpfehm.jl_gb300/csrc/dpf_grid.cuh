// dpf_grid.cuh -- the barrier of the persistent solve kernels, between all blocks of a cooperative
// launch (one block per SM, so all of them are resident).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dpf {

// Two counters 128 bytes apart: arrivals, and the last barrier whose last() is done. Zeroed before a launch.
constexpr int kGridBarWords = 64;
constexpr uint64_t kGridWaitNs = 1000000000ull;  // a wait ends after one second ...
constexpr uint32_t kGridWaitTries = 1u << 28;    // ... or, should the global timer stall, 2^28 polls

// Every thread of every block calls sync(last) the same number of times. The last block to arrive runs
// last() (all its threads) before the others go on: the reductions of a phase are finished there, so
// they need no barrier of their own. False (in every thread of the block) when the wait ran out: the
// error word is set and the kernel returns; the other blocks' waits run out the same way. The limit is wall time: it
// also runs out where other work holds the SMs that the missing blocks wait for, or a phase of the solve itself
// takes longer. The host then finishes the solve with the separate kernels, in which no block waits for another.
struct GridBar {
    unsigned *words;
    int *err;
    unsigned gen = 0;

    // Polls *word until it reaches `to`, which makes the other blocks' writes visible to this block. Every
    // poll is an acquire: with relaxed polls and an acquire fence behind them a barrier between a write and a
    // read by all threads took 0.2 us more (2.10 -> 1.89 us with its accesses; 1024 threads on 152 SMs). Eight
    // arrival counters (2.25 us), a flag per block polled by a warp (3.4 us) and a last arriver that sets a
    // separate word (2.4 us) were slower.
    __device__ __forceinline__ bool wait(const unsigned *word, unsigned to) {
        uint64_t t0 = 0;
        bool got = true;
        for (uint32_t k = 0;; k++) {
            unsigned seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(word) : "memory");
            if ((int)(seen - to) >= 0) break;
            if ((k & 63) == 63) {
                uint64_t t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                if (t - t0 > kGridWaitNs || k >= kGridWaitTries) {
                    atomicExch(err, 1);
                    got = false;
                    break;
                }
            }
        }
        return got;
    }
    // without a last(): the arrivals themselves are polled, one trip to L2 less (2.5 -> 1.4 us)
    __device__ __forceinline__ bool sync() {
        __shared__ int ok;
        __syncthreads();  // the block's work of this phase is issued
        gen++;
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(words) : "memory");
            ok = wait(words, gen * gridDim.x);
        }
        __syncthreads();
        return ok != 0;
    }
    template <typename F>
    __device__ __forceinline__ bool sync(F last) {
        __shared__ int arrived_last, ok;
        __syncthreads();
        gen++;
        if (threadIdx.x == 0) {
            unsigned before;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(words) : "memory");
            arrived_last = before + 1u == gen * gridDim.x;
            ok = 1;
            if (!arrived_last) ok = wait(words + 32, gen);
        }
        __syncthreads();
        if (arrived_last) {
            last();
            __syncthreads();
            if (threadIdx.x == 0)
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(words + 32), "r"(gen) : "memory");
        }
        return ok != 0;
    }
};

}  // namespace dpf
