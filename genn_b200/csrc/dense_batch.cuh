// DENSE delivery of a batched network: every weight row that a step needs is read once for all the copies that need it.
//
// The rows are what bounds it.  With 32 copies at 2.5 % a step reaches 55 % of the rows, 1.44 copies each; one pass over the
// rows per copy (presynapticPostSpanKernel) moves 1.44 times the bytes, and its threads wait for one load after another.
// Here a CTA owns DENSE_COLS columns and a range of source neurons.  It turns the copies' spike lists into one bit mask per
// source neuron (bit b: copy b spiked) and gathers the sources that have one into a list.  The listed rows pass through a
// ring of DENSE_STAGES stages of 32 rows in shared memory (two CTAs on an SM: 128 KB under way, several times what HBM's
// latency wants); one warp sends for them, a row a lane, as bulk copies, and the others fall behind one another by as much
// as the ring holds (with a barrier per stage every stage took as long as its busiest warp).  A warp owns copies: a ballot
// over the masks of a stage's rows gives the rows its copy needs, which it sums in registers, so that sums cost neither
// shared memory nor atomics until one 16-byte reduction per four columns at the end.  Sums in shared
// memory, the masks' bits walked row by row, took 55 us at the size below, stages of half the columns brought in by all
// threads 42, eight adding warps 33; now DRAM stands at two thirds of a copy's rate and the issue slots at 43 %.
//
// 8192 x 8192, 32 copies, 25 Hz at 1 ms (149 MB of rows a step): 107 us with presynapticPostSpanKernel, 31 here (a step with the neuron
// update 36.5).
#pragma once

#include "common.cuh"
#include "presynaptic_update.cuh"

namespace b200
{
constexpr unsigned int DENSE_WARPS = 16;            // warps that add; one more brings the rows in
constexpr unsigned int DENSE_BLOCK = DENSE_WARPS * 32 + 32;
constexpr unsigned int DENSE_COLS = 256;            // columns of a CTA: twice four a lane
constexpr unsigned int DENSE_COPIES = 32;           // copies of a CTA: one mask word
constexpr unsigned int DENSE_OWN = DENSE_COPIES / DENSE_WARPS;      // copies of a warp
constexpr unsigned int DENSE_STAGES = 3;
constexpr unsigned int DENSE_PER_SM = 2;            // CTAs on an SM: 96 KB of stages each
constexpr unsigned int DENSE_WINDOW = 1024;         // most source neurons of a CTA (masks and list: 6 KB)
// (There is no upper limit: every CTA reads all spike lists to find its own sources, but 100 000 x 512 with 2 / 8 / 32 copies takes 25 / 26
// / 59 us a step at 20 Hz, 400 000 x 128 81 / 97 / 219, where the kernel with a thread per column takes 468 / 491 / 536 and 1842
// / 1942 / 2189.)
// With fewer sources a thread per column that walks a copy's few spikes one after another is done before the masks are made:
// a step of 2 / 8 / 32 copies takes 7.7 / 7.7 / 8.6 us with it and 7.9 / 8.4 / 9.7 here at 600 x 2400, but 9.1 / 9.6 / 10.2
// against 7.6 / 8.3 / 9.9 at 1200 x 1200 and 12.9 / 13.3 / 14.2 against 7.7 / 8.3 / 9.6 at 2400 x 600.
constexpr unsigned int DENSE_LEAST_SOURCES = 1024;

struct DenseLaunch
{
    SynapseLaunch S;                    // DENSE groups that do not learn
    const uint4 *parts;                 // per CTA: group, first column, first source, number of sources
};

constexpr size_t DENSE_SMEM = DENSE_STAGES * 32 * DENSE_COLS * sizeof(float) + DENSE_WINDOW * (sizeof(unsigned int) + sizeof(uint16_t));

__device__ __forceinline__ unsigned int denseShare(const void *p) { return (unsigned int)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void denseSum(float4 &sum, const float4 &v)
{
    sum.x = B200_FADD(sum.x, v.x); sum.y = B200_FADD(sum.y, v.y);
    sum.z = B200_FADD(sum.z, v.z); sum.w = B200_FADD(sum.w, v.w);
}

static __global__ void __launch_bounds__(DENSE_BLOCK, DENSE_PER_SM)
denseBatchKernel(const DenseLaunch L)
{
    extern __shared__ __align__(16) unsigned char denseShared[];
    __shared__ unsigned int listed;
    __shared__ __align__(8) unsigned long long arrived[DENSE_STAGES], released[DENSE_STAGES];
    const uint4 part = __ldg(&L.parts[blockIdx.x]);
    __shared__ __align__(16) b200_synapse_group g;
    stageGroup(g, L.S.groups[part.x]);
    const unsigned int firstCopy = blockIdx.z * DENSE_COPIES, copies = min(DENSE_COPIES, L.S.batch - firstCopy);
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned int rowStride = g.num_trg, cols = min(DENSE_COLS, rowStride - part.y);
    const bool vec = (rowStride & 3u) == 0u && ((reinterpret_cast<size_t>(g.g) | reinterpret_cast<size_t>(g.out_post)) & 15u) == 0u;    // rows keep a 16-byte alignment
    const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    float *const stages = reinterpret_cast<float*>(denseShared);
    unsigned int *const mask = reinterpret_cast<unsigned int*>(stages + DENSE_STAGES * 32u * DENSE_COLS);
    uint16_t *const list = reinterpret_cast<uint16_t*>(mask + DENSE_WINDOW);
    if(threadIdx.x == 0u) {
        listed = 0u;
        // a stage is complete when its bytes are: the sending warp's first lane announces them, or its lanes' copies arrive
        for(unsigned int i = 0; i < DENSE_STAGES; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(denseShare(&arrived[i])), "r"(vec ? 1u : 32u) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(denseShare(&released[i])), "r"(DENSE_WARPS) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for(unsigned int i = threadIdx.x; i < part.w; i += DENSE_BLOCK) mask[i] = 0u;
    __syncthreads();
    chainWait();
    const unsigned int k = chainPhase(L.S.state, L.S.ahead), polls = L.S.state->copy_wait_limit;
    const unsigned int slots = g.src_delay_slots, slot = ringSlot(k + slots - g.axonal_delay, slots);

    // ---- spike lists -> masks of this CTA's sources: the lists of a warp's copies side by side
    if(warp < DENSE_WARPS) {
        const unsigned int *spk[DENSE_OWN];
        unsigned int n[DENSE_OWN], most = 0u;
        #pragma unroll
        for(unsigned int o = 0; o < DENSE_OWN; o++) {
            const unsigned int b = warp + o * DENSE_WARPS;
            spk[o] = g.src_spk + ((unsigned long long)(firstCopy + b) * slots + slot) * g.num_src;
            n[o] = b < copies ? min(g.src_spk_cnt[(firstCopy + b) * slots + slot], g.num_src) : 0u;
        }
        #pragma unroll
        for(unsigned int o = 0; o < DENSE_OWN; o++) most = max(most, n[o]);
        for(unsigned int at = lane; at < most; at += 32u * 4u) {
            unsigned int id[DENSE_OWN][4];
            #pragma unroll
            for(unsigned int o = 0; o < DENSE_OWN; o++) {
                #pragma unroll
                for(unsigned int j = 0; j < 4u; j++) id[o][j] = (at + 32u * j < n[o]) ? spk[o][at + 32u * j] : 0xFFFFFFFFu;
            }
            #pragma unroll
            for(unsigned int o = 0; o < DENSE_OWN; o++) {
                #pragma unroll
                for(unsigned int j = 0; j < 4u; j++) {
                    if(id[o][j] - part.z < part.w) atomicOr(&mask[id[o][j] - part.z], 1u << (warp + o * DENSE_WARPS));
                }
            }
        }
        unsigned long long spikes = 0;
        #pragma unroll
        for(unsigned int o = 0; o < DENSE_OWN; o++) spikes += n[o];
        if(L.S.count_events && part.y == 0u && part.z == 0u && lane == 0u) {
            atomicAdd(&L.S.state->synaptic_events, spikes * g.num_trg);
        }
    }
    __syncthreads();
    for(unsigned int i = threadIdx.x; i < ((part.w + 31u) & ~31u); i += DENSE_BLOCK) {
        const bool any = i < part.w && mask[i] != 0u;
        const unsigned int ballot = __ballot_sync(0xFFFFFFFFu, any);
        unsigned int base = 0;
        if(lane == 0u && ballot) base = atomicAdd(&listed, (unsigned int)__popc(ballot));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if(any) list[base + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)i;
    }
    __syncthreads();
    const unsigned int rows = listed;
    if(rows == 0u) return;

    // ---- rows through the ring
    const float *const base = constant ? nullptr : g.g + (unsigned long long)part.z * rowStride + part.y;
    const unsigned int numStages = constant ? 0u : (rows + 31u) / 32u;
    if(warp == DENSE_WARPS) {
        unsigned int stage = 0;
        // Rows leave L2 before anything else does: the neurons' state, which the next kernel reads, stays there (8192 x 8192, 32
        // copies: a step with the neuron update 39.1 -> 37.3 us; keeping an eighth, a quarter, half or all of the rows instead 37.0, 37.1, 37.9, 39.2)
        unsigned long long soon;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(soon));
        for(; stage < numStages; stage++) {
            const unsigned int ring = stage % DENSE_STAGES;
            if(stage >= DENSE_STAGES && !__all_sync(0xFFFFFFFFu, copyArrived(&released[ring], (stage / DENSE_STAGES - 1u) & 1u, polls))) {
                if(lane == 0u) atomicOr(&L.S.state->error, ERR_COPY_TIMEOUT);
                break;
            }
            float *const to = stages + ring * 32u * DENSE_COLS;
            const unsigned int n = min(32u, rows - stage * 32u), bar = denseShare(&arrived[ring]);
            if(vec) {
                if(lane == 0u) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(n * cols * 4u) : "memory");
                __syncwarp();
                if(lane < n) {
                    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                                 :: "r"(denseShare(to + lane * DENSE_COLS)), "l"(__cvta_generic_to_global(base + (unsigned long long)list[stage * 32u + lane] * rowStride)),
                                    "r"(cols * 4u), "r"(bar), "l"(soon) : "memory");
                }
            }
            else {
                for(unsigned int j = 0; j < n; j++) {
                    const float *const row = base + (unsigned long long)list[stage * 32u + j] * rowStride;
                    for(unsigned int col = lane; col < cols; col += 32u) {
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(denseShare(to + j * DENSE_COLS + col)), "l"(__cvta_generic_to_global(row + col)) : "memory");
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(bar) : "memory");
            }
        }
        // (the others wait for every stage too, unless they have given up)
        for(unsigned int sent = stage > DENSE_STAGES ? stage - DENSE_STAGES : 0u; sent < stage; sent++) {
            copyArrived(&arrived[sent % DENSE_STAGES], (sent / DENSE_STAGES) & 1u, COPY_WAITS);
        }
        return;
    }
    // fewer copies than warps: several warps share a copy, each with every `sharers`-th row
    const unsigned int sharers = copies >= DENSE_WARPS ? 1u : DENSE_WARPS / copies, share = copies >= DENSE_WARPS ? 0u : warp / copies;
    const unsigned int first = copies >= DENSE_WARPS ? warp : warp % copies;
    const bool mine = share < sharers && (lane % sharers) == share;
    float4 sum[DENSE_OWN][2];
    #pragma unroll
    for(unsigned int o = 0; o < DENSE_OWN; o++) sum[o][0] = sum[o][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    unsigned int ring = 0, parity = 0;
    for(unsigned int stage = 0; stage < numStages; stage++) {
        const bool there = copyArrived(&arrived[ring], parity, polls);
        const unsigned int at = stage * 32u + lane;
        const unsigned int m = (mine && there && at < rows) ? mask[list[at]] >> first : 0u;
        const float4 *const w = reinterpret_cast<const float4*>(stages + ring * 32u * DENSE_COLS) + lane;
        #pragma unroll
        for(unsigned int o = 0; o < DENSE_OWN; o++) {
            // two rows at a time: the loads of one behind the other's
            unsigned int left = __ballot_sync(0xFFFFFFFFu, (m >> (o * DENSE_WARPS)) & 1u);
            while(left) {
                const float4 *const row = w + (31 - __clz(left)) * (DENSE_COLS / 4u);
                left ^= 0x80000000u >> __clz(left);
                const float4 v0 = row[0], v1 = row[32];
                if(left) {
                    const float4 *const next = w + (31 - __clz(left)) * (DENSE_COLS / 4u);
                    left ^= 0x80000000u >> __clz(left);
                    const float4 u0 = next[0], u1 = next[32];
                    denseSum(sum[o][0], v0);
                    denseSum(sum[o][1], v1);
                    denseSum(sum[o][0], u0);
                    denseSum(sum[o][1], u1);
                }
                else {
                    denseSum(sum[o][0], v0);
                    denseSum(sum[o][1], v1);
                }
            }
        }
        // the lanes' vote after the stage, not before it: each waits for itself
        if(!__all_sync(0xFFFFFFFFu, there)) {
            if(lane == 0u) atomicOr(&L.S.state->error, ERR_COPY_TIMEOUT);
            return;
        }
        __syncwarp();
        if(lane == 0u) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(denseShare(&released[ring])) : "memory");
        if(++ring == DENSE_STAGES) {
            ring = 0;
            parity ^= 1u;
        }
    }
    if(constant) {
        // nothing to read: every listed row adds the same weight
        const float c = g.wu_params[0];
        for(unsigned int at = lane; at < ((rows + 31u) & ~31u); at += 32u) {
            const unsigned int m = (mine && at < rows) ? mask[list[at]] >> first : 0u;
            #pragma unroll
            for(unsigned int o = 0; o < DENSE_OWN; o++) {
                for(unsigned int n = __popc(__ballot_sync(0xFFFFFFFFu, (m >> (o * DENSE_WARPS)) & 1u)); n; n--) {
                    denseSum(sum[o][0], make_float4(c, c, c, c));
                }
                sum[o][1] = sum[o][0];
            }
        }
    }

    // ---- the sums, out to the targets' input
    #pragma unroll
    for(unsigned int o = 0; o < DENSE_OWN; o++) {
        #pragma unroll
        for(unsigned int half = 0; half < 2u; half++) {
            const unsigned int b = first + o * DENSE_WARPS, col = half * 128u + lane * 4u;
            const float4 a = sum[o][half];
            if(b >= copies || share >= sharers || col >= cols || (a.x == 0.0f && a.y == 0.0f && a.z == 0.0f && a.w == 0.0f)) continue;
            float *const out = g.out_post + (unsigned long long)(firstCopy + b) * g.num_trg + part.y + col;
            if(vec) redAdd4(out, a);
            else {
                redAdd(out, a.x);
                if(col + 1u < cols) redAdd(out + 1, a.y);
                if(col + 2u < cols) redAdd(out + 2, a.z);
                if(col + 3u < cols) redAdd(out + 3, a.w);
            }
        }
    }
}
}   // namespace b200
