// dp_barrier.cuh - the bounded grid barrier of the persistent kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gqb {

constexpr unsigned long long kBarrierTimeoutNs = 4000000000ull;   // 4 s of global time
constexpr unsigned kBarrierSpinLimit = 1u << 26;                  // hard cap on polls as well (~30 s)

// poll limit of one barrier wait: the launch argument when non-zero (the
// gpuqo_b200_barrier_poll_limit setting, which makes waits run out on purpose
// so that the timeout path can be exercised), else kBarrierSpinLimit
__device__ __forceinline__ unsigned barrier_polls(unsigned poll_limit) {
    return poll_limit != 0u ? poll_limit : kBarrierSpinLimit;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// bar[0] = arrivals (base at launch), bar[2] = error flag (zero at launch).
// The arrival counter only grows: a block's e-th barrier of the launch
// completes when it reaches base + e * gridDim.x, so nobody resets it, the last
// block to arrive has nothing more to do, and the next launch may go on from
// where it stands.  Thread 0 arrives with a gpu-scope release reduction
// (ordering every write its block made before the __syncthreads) and polls
// with gpu-scope acquire loads (ACQUIRE_POLL), or with relaxed loads and one
// fence once the count is reached: an acquire load also drops the SM's L1
// contents, which a kernel that keeps its working data in shared memory does
// not mind (k_dp_tree: the faster barrier) but which costs the batch kernel,
// whose per-query data is read through L1 while waiting blocks poll on the
// same SM.  The verdict is the same for every thread of the block (thread 0
// decides); blocks may disagree only after a timeout, and then every later
// barrier sees the error flag and returns false at once, so all blocks leave.
// A poll is one round trip to L2 (some 700 cycles); the error flag comes with
// it, because a second trip for the flag after the count, and a third for the
// verdict, would lengthen every level by half a microsecond.
// epoch: the caller's count of barriers passed (thread 0); max_polls: polls
// before the wait gives up (barrier_polls).
template <bool ACQUIRE_POLL>
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned &epoch, unsigned max_polls, unsigned base = 0u) {
    __shared__ unsigned s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        epoch++;
        const unsigned target = base + epoch * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        const unsigned long long t0 = global_ns();
        unsigned spins = 0, failed;
        for (;;) {
            // error flag and count in flight together
            unsigned c;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(failed) : "l"(bar + 2) : "memory");
            if (ACQUIRE_POLL) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
            } else {
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
            }
            if (c >= target || failed != 0u) {
                if (!ACQUIRE_POLL) __threadfence();
                break;
            }
            ++spins;
            if (spins >= max_polls || ((spins & 63u) == 0u && global_ns() - t0 > kBarrierTimeoutNs)) {
                atomicExch(bar + 2, 1u);
                failed = 1u;
                break;
            }
        }
        s_ok = failed == 0u ? 1u : 0u;
    }
    __syncthreads();
    return s_ok != 0u;
}

// The barrier of a grid that is one thread-block cluster, in hardware (no
// polling, nothing to time out): every thread of the cluster.  It follows
// code in which single lanes write a set's winner or emit a list's entries, so
// a warp may arrive in parts: the forms without .aligned, which every thread
// executes for itself.
__device__ __forceinline__ uint32_t cluster_blocks() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace gqb
