// Shared device-side definitions for the sm_100a kernel templates.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "genn_b200.h"
#include "genn_b200_rng.h"

namespace b200
{
// Step counters kept on the device so a captured step graph can be replayed
// without touching kernel arguments: `timestep` gives t = timestep * dt,
// `steps_done` drives every ring pointer (spike queue slot, dendritic-delay
// front), `ticket` elects the last block of the neuron kernel, `error` is set
// by bounds checks.
struct StepState
{
    unsigned long long timestep;
    unsigned long long steps_done;
    unsigned int ticket;
    unsigned int error;
    // steps_done modulo ring_period, a common multiple of every ring size (spike
    // queue depths, dendritic-delay depths), so ring slots come from 32-bit
    // arithmetic: (phase + c) % n == (steps_done + c) % n for every ring size n
    unsigned int phase;
    unsigned int ring_period;
    unsigned long long synaptic_events;   // only advanced when event counting is on
    unsigned long long spikes;
    // SM clock cycles CTA 0 spent in each phase of the persistent kernel:
    // presynaptic work, barrier after it, neuron work, barrier after it
    unsigned long long phase_cycles[4];
    unsigned long long probe[12];        // finer clock64 sums of the persistent kernel's profile mode
    // verdict of tiledDecideKernel for the step being delivered: 1 = enough events for the
    // target-tiled kernel, 0 = the one-reduction-per-event kernel delivers
    unsigned int heavy;
    // most spikes (all populations and batch entries together) any step has emitted since the host last
    // read and cleared this word: tells the host whether launching the tiled kernels is worth it at all
    unsigned int peak_spikes;
    // limits of every wait inside the persistent kernels (set by the host; a wait that runs out sets an
    // error bit, all CTAs leave the kernel and the host reports it): polls of the grid barrier, polls for
    // a word another process writes, SM cycles a warp waits for work from another warp of its CTA
    unsigned long long barrier_spin_limit;
    unsigned long long exchange_spin_limit;
    long long stream_wait_cycles;
    // polls for a copy into shared memory (dense_batch.cuh, sparse_batch.cuh)
    unsigned int copy_wait_limit;
    // target-resident kernel (resident.h: "Busy networks"): what it has lost to the kernel with a grid barrier (ns), the step
    // until which that one goes on in its place, and for how many steps it last did
    unsigned int resident_debt;
    unsigned int resident_rest;
    unsigned long long resident_hold;
};

constexpr unsigned int ERR_SPIKE_OVERFLOW = 1u;
constexpr unsigned int ERR_IND_RANGE = 2u;
constexpr unsigned int ERR_DELAY_RANGE = 4u;
constexpr unsigned int ERR_BARRIER_TIMEOUT = 8u;
constexpr unsigned int ERR_COPY_TIMEOUT = 64u;          // (32: ERR_EXCHANGE_TIMEOUT)

// Polls for a copy into shared memory, unless the host set another limit.  A kernel that gives up waits, this long again, for what
// it has sent for: nothing may arrive in a block's shared memory after the block.
constexpr unsigned int COPY_WAITS = 1u << 18;

// Waits for a phase of a shared-memory barrier.
__device__ __forceinline__ bool copyArrived(const unsigned long long *bar, unsigned int parity, unsigned int polls)
{
    for(unsigned int i = 0; i < polls; i++) {
        unsigned int done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"((unsigned int)__cvta_generic_to_shared(bar)), "r"(parity) : "memory");
        if(done) return true;
    }
    return false;
}

// Block -> merged-group element lookup: block_start[g] is the first block of
// group g, block_start[num_groups] the grid size.  Linear for a handful of
// groups, binary beyond that (the reference emits the same two forms,
// backendSIMT.h:244-323).
__device__ __forceinline__ unsigned int findGroup(const unsigned int *__restrict__ block_start,
                                                  unsigned int num_groups, unsigned int block)
{
    // plain loads: the table may live in shared memory
    if(num_groups <= 8) {
        unsigned int g = 0;
        while(g + 1 < num_groups && block >= block_start[g + 1]) g++;
        return g;
    }
    unsigned int lo = 0, hi = num_groups;
    while(hi - lo > 1) {
        const unsigned int mid = (lo + hi) >> 1;
        if(block >= block_start[mid]) lo = mid; else hi = mid;
    }
    return lo;
}

// fp32 add to GLOBAL memory with no return value.  The address space is spelled out: after a
// reduction through a generic pointer the load/store unit holds back later generic accesses
// (the staged tables in shared memory are read through generic pointers) until it completes.
__device__ __forceinline__ void redAdd(float *addr, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" :: "l"(__cvta_generic_to_global(addr)), "f"(v));
}

// Four neighbouring cells at once (16-byte aligned).
__device__ __forceinline__ void redAdd4(float *addr, const float4 &v)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" :: "l"(__cvta_generic_to_global(addr)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
}

// The kernels of the one-launch-per-kernel path follow one another as dependent launches: a kernel's blocks may be placed,
// and read what no kernel writes, while the kernel before it still runs; chainWait() holds them until that one's results
// are there.  Every kernel says at once that the next one may be placed: nothing of it runs past its own chainWait().
__device__ __forceinline__ void chainWait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A block of steps advances the counters once, with its last kernel; the kernels of its step number `ahead` count for
// themselves (an election of a last block in every step cost 2 us a step).
__device__ __forceinline__ unsigned int chainPhase(const StepState *state, unsigned int ahead)
{
    unsigned int k = state->phase + ahead;
    const unsigned int period = state->ring_period;
    if(k >= period && period) k %= period;
    return k;
}

__device__ __forceinline__ unsigned int ringSlot(unsigned int k, unsigned int slots)
{
    return k % slots;
}

// Copy `bytes` (a multiple of 4) from global to shared memory with the whole CTA.
__device__ __forceinline__ void stageWords(void *dst, const void *src, size_t bytes)
{
    unsigned int *d = static_cast<unsigned int*>(dst);
    const unsigned int *s = static_cast<const unsigned int*>(src);
    for(size_t w = threadIdx.x; w < bytes / 4; w += blockDim.x) d[w] = __ldg(&s[w]);
}

// What a kernel needs of its group, into shared memory ahead of chainWait(): nothing writes a group's table while kernels run, and read
// behind the wait every field that leads to an address cost another round trip to memory.  A step of DENSE 1200 x 1200 with 8 copies:
// 8.25 -> 7.00 us (the DENSE kernel and the neuron update), of 5000 + 5000 neurons with 3 copies 9.18 -> 8.81.  (Shared memory is
// not free in kernels that use little else of it: neuronStaged.)
template<typename T>
__device__ __forceinline__ void stageGroup(T &shared, const T &group)
{
    stageWords(&shared, &group, sizeof(T));
    __syncthreads();
}

// The same without waiting: several tables take one round trip to memory, not one each.  stagedWords() and a barrier of the CTA
// end it.
__device__ __forceinline__ void stageWordsAsync(void *dst, const void *src, size_t bytes)
{
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
    const unsigned int *s = static_cast<const unsigned int*>(src);
    for(unsigned int w = threadIdx.x; w < (unsigned int)(bytes / 4); w += blockDim.x) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(d + 4u * w), "l"(__cvta_generic_to_global(s + w)) : "memory");
    }
}

__device__ __forceinline__ void stagedWords()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }
}   // namespace b200
