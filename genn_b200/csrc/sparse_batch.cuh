// SPARSE delivery of a batched network whose target buffers fit an SM's shared memory.
//
// One reduction into L2 per synaptic event is bound by the 1.9e11 scattered reductions a second that the L2 takes (measured;
// 11 M events: 59 us), one addition in shared memory by 8e11.  A CTA takes one copy of one target buffer (outPost, or a whole
// dendritic-delay ring) into its shared memory as private sums, a share of that copy's spikes, and adds their rows as they
// lie in the model's arrays: whole rows, 6 to 9 bytes a synapse, no second copy of the synapses and no table of runs.  The
// sums go to the target once at the end, 16 bytes a reduction.  A share with few events (SCATTER_FEW) leaves the sums alone
// and reduces straight into L2: clearing and flushing them would take longer.
//
// Shares: the spikes of all groups onto the buffer stand on one line, each as long as its group's rows; a CTA owns an equal
// stretch of the line and computes it from the spike counts itself.  Inside, a warp takes pieces of SCATTER_PIECE synapses,
// the next piece's loads under way while one is added (a piece is 8 bytes of weight and index a lane and load; 32 warps with
// two pieces in flight keep 50 KB under way on an SM, about what HBM needs).
//
// 20 000 + 20 000 neurons, 8 copies, 11 M events a step: 90 us with the tiled kernels, 60 here.
#pragma once

#include "common.cuh"
#include "presynaptic_update.cuh"

namespace b200
{
constexpr unsigned int SCATTER_BLOCK = 1024;
constexpr unsigned int SCATTER_WARPS = SCATTER_BLOCK / 32;
constexpr unsigned int SCATTER_QUADS = 2;                               // groups of four synapses of a lane in a piece
constexpr unsigned int SCATTER_PIECE = 32 * 4 * SCATTER_QUADS;
constexpr unsigned int SCATTER_MOST_CELLS = 52 * 1024;                  // 208 KB of sums
constexpr unsigned int SCATTER_MOST_SOURCES = 64;                       // groups onto one buffer
// An event costs 0.19 ns of an SM's shared memory and 0.78 ns of its share of the L2's reductions; clearing and flushing
// the sums about 2.5 us.
constexpr unsigned int SCATTER_FEW = 4096;

struct ScatterTarget
{
    float *cells;                       // copy 0 of the buffer
    unsigned int num_cells;             // of one copy: targets, or ring slots x targets
    unsigned int first_group;           // groups of the table that deliver here
    unsigned int num_groups;
};

struct ScatterPart                      // what a CTA does
{
    unsigned int target, copy, share, shares;
};

struct ScatterLaunch
{
    SynapseLaunch S;                    // SPARSE groups that do not learn, in the order of their targets
    const ScatterTarget *targets;
    const ScatterPart *parts;
};

__device__ __forceinline__ void scatterShared(float *cell, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;" :: "r"((unsigned int)__cvta_generic_to_shared(cell)), "f"(v) : "memory");
}

// Four synapses as they are stored.
struct ScatterQuad
{
    uint4 ind;
    float4 w;
    unsigned int delay;
};

// One piece of a spike's row between its loads and its additions.
struct ScatterHeld
{
    ScatterQuad quad[SCATTER_QUADS];
    unsigned int length, pre, piece;    // length 0: nothing
};

__device__ __forceinline__ void scatterFetch(const b200_synapse_group &g, ScatterHeld &h, unsigned int lane)
{
    const unsigned long long rowStart = (unsigned long long)h.pre * g.row_stride, all = (unsigned long long)g.num_src * g.row_stride;
    const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    h.length = __ldg(&g.row_length[h.pre]);
    #pragma unroll
    for(unsigned int q = 0; q < SCATTER_QUADS; q++) {
        // quads are aligned to the array, not to the row; past the end of the row they still lie in the array or its padding
        const unsigned long long idx = (rowStart & ~3ull) + (unsigned long long)h.piece * SCATTER_PIECE + (q * 32u + lane) * 4u;
        ScatterQuad &Q = h.quad[q];
        if(idx >= all) continue;
        if(g.ind_bytes == 2u) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(g.ind) + idx));
            Q.ind.x = v.x; Q.ind.y = v.y;
        }
        else if(g.ind_bytes == 4u) Q.ind = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint32_t*>(g.ind) + idx));
        else Q.ind.x = __ldg(reinterpret_cast<const unsigned int*>(static_cast<const uint8_t*>(g.ind) + idx));
        if(!constant) Q.w = __ldg(reinterpret_cast<const float4*>(g.g + idx));
        if(g.max_den_delay) Q.delay = __ldg(reinterpret_cast<const unsigned int*>(g.d + idx));
    }
}

__device__ __forceinline__ void scatterAdd(const b200_synapse_group &g, const ScatterHeld &h, float *sums, float *cells, bool few,
                                           unsigned int front, unsigned int lane, StepState *state)
{
    const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    const unsigned int skew = (unsigned int)(((unsigned long long)h.pre * g.row_stride) & 3ull);
    const unsigned int D = g.max_den_delay, numTrg = g.num_trg, end = skew + h.length;
    #pragma unroll
    for(unsigned int q = 0; q < SCATTER_QUADS; q++) {
        const ScatterQuad &Q = h.quad[q];
        const unsigned int at = h.piece * SCATTER_PIECE + (q * 32u + lane) * 4u;
        if(at >= end) continue;
        unsigned int post[4];
        if(g.ind_bytes == 2u) {
            post[0] = Q.ind.x & 0xFFFFu; post[1] = Q.ind.x >> 16; post[2] = Q.ind.y & 0xFFFFu; post[3] = Q.ind.y >> 16;
        }
        else if(g.ind_bytes == 4u) {
            post[0] = Q.ind.x; post[1] = Q.ind.y; post[2] = Q.ind.z; post[3] = Q.ind.w;
        }
        else {
            post[0] = Q.ind.x & 0xFFu; post[1] = (Q.ind.x >> 8) & 0xFFu; post[2] = (Q.ind.x >> 16) & 0xFFu; post[3] = Q.ind.x >> 24;
        }
        const float w[4] = {Q.w.x, Q.w.y, Q.w.z, Q.w.w};
        #pragma unroll
        for(unsigned int j = 0; j < 4u; j++) {
            if(at + j < skew || at + j >= end) continue;
            unsigned int cell = post[j];
            if(cell >= numTrg) {
                atomicOr(&state->error, ERR_IND_RANGE);
                continue;
            }
            if(D) {
                unsigned int slot = front + ((Q.delay >> (8u * j)) & 0xFFu);
                while(slot >= D) slot -= D;
                cell += slot * numTrg;
            }
            const float v = constant ? g.wu_params[0] : w[j];
            if(few) redAdd(cells + cell, v);
            else scatterShared(sums + cell, v);
        }
    }
}

static __global__ void __launch_bounds__(SCATTER_BLOCK, 1)
sparseBatchKernel(const ScatterLaunch L)
{
    extern __shared__ __align__(16) float scatterSums[];
    __shared__ unsigned int firstSpike[SCATTER_MOST_SOURCES], spikes[SCATTER_MOST_SOURCES];
    __shared__ unsigned long long line[SCATTER_MOST_SOURCES];
    const ScatterPart part = L.parts[blockIdx.x];
    const ScatterTarget T = L.targets[part.target];
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    chainWait();
    const unsigned int k = chainPhase(L.S.state, L.S.ahead);
    // ---- this CTA's stretch of the line of spikes
    if(threadIdx.x < T.num_groups) {
        const b200_synapse_group &g = L.S.groups[T.first_group + threadIdx.x];
        const unsigned int slots = g.src_delay_slots, slot = ringSlot(k + slots - g.axonal_delay, slots);
        spikes[threadIdx.x] = min(g.src_spk_cnt[part.copy * slots + slot], g.num_src);
        line[threadIdx.x] = (unsigned long long)spikes[threadIdx.x] * g.row_stride;
    }
    __syncthreads();
    unsigned long long all = 0, before = 0;
    for(unsigned int i = 0; i < T.num_groups; i++) {
        all += line[i];
        if(i < threadIdx.x) before += line[i];
    }
    const unsigned long long low = all * part.share / part.shares, high = all * (part.share + 1u) / part.shares;
    if(low == high) return;
    const bool few = high - low < SCATTER_FEW;
    __syncthreads();
    if(threadIdx.x < T.num_groups) {
        // spike i of a group stands at `before` + i * row_stride
        const unsigned int stride = max(1u, L.S.groups[T.first_group + threadIdx.x].row_stride);
        auto from = [&](unsigned long long at) {
            return at <= before ? 0u : (unsigned int)min((unsigned long long)spikes[threadIdx.x], (at - before + stride - 1u) / stride);
        };
        const unsigned int first = from(low);
        firstSpike[threadIdx.x] = first;
        spikes[threadIdx.x] = from(high) - first;
    }
    if(!few) {
        for(unsigned int i = threadIdx.x; i < (T.num_cells + 3u) / 4u; i += SCATTER_BLOCK) {
            reinterpret_cast<float4*>(scatterSums)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    __syncthreads();
    float *const cells = T.cells + (unsigned long long)part.copy * T.num_cells;
    unsigned int item = warp;
    for(unsigned int gi = 0; gi < T.num_groups; gi++) {
        const b200_synapse_group &g = L.S.groups[T.first_group + gi];
        const unsigned int pieces = (g.row_stride + 3u + SCATTER_PIECE - 1u) / SCATTER_PIECE, items = spikes[gi] * pieces;
        const unsigned int slots = g.src_delay_slots, slot = ringSlot(k + slots - g.axonal_delay, slots);
        const unsigned int *const spk = g.src_spk + ((unsigned long long)part.copy * slots + slot) * g.num_src + firstSpike[gi];
        const unsigned int front = g.max_den_delay ? ringSlot(k + 1u, g.max_den_delay) : 0u;
        auto spikeOf = [&](unsigned int at) { return at < items ? spk[at / pieces] : 0u; };
        auto fetch = [&](ScatterHeld &h, unsigned int at, unsigned int pre) {
            h.length = 0u;
            if(at >= items) return;
            if(pre >= g.num_src) {
                atomicOr(&L.S.state->error, ERR_IND_RANGE);
                return;
            }
            h.pre = pre;
            h.piece = at % pieces;
            scatterFetch(g, h, lane);
            if(L.S.count_events && h.piece == 0u && lane == 0u) atomicAdd(&L.S.state->synaptic_events, (unsigned long long)h.length);
        };
        ScatterHeld a, b;
        fetch(a, item, spikeOf(item));
        unsigned int next = spikeOf(item + SCATTER_WARPS);
        while(item < items) {
            fetch(b, item + SCATTER_WARPS, next);
            next = spikeOf(item + 2u * SCATTER_WARPS);
            scatterAdd(g, a, scatterSums, cells, few, front, lane, L.S.state);
            item += SCATTER_WARPS;
            if(item >= items) break;
            fetch(a, item + SCATTER_WARPS, next);
            next = spikeOf(item + 2u * SCATTER_WARPS);
            scatterAdd(g, b, scatterSums, cells, few, front, lane, L.S.state);
            item += SCATTER_WARPS;
        }
        item -= items;
    }
    if(few) return;
    __syncthreads();
    if((T.num_cells & 3u) == 0u) {
        for(unsigned int i = threadIdx.x; i < T.num_cells / 4u; i += SCATTER_BLOCK) {
            const float4 a = reinterpret_cast<const float4*>(scatterSums)[i];
            if(a.x != 0.0f || a.y != 0.0f || a.z != 0.0f || a.w != 0.0f) redAdd4(cells + 4u * i, a);
        }
    }
    else {
        for(unsigned int i = threadIdx.x; i < T.num_cells; i += SCATTER_BLOCK) {
            if(scatterSums[i] != 0.0f) redAdd(cells + i, scatterSums[i]);
        }
    }
}
}   // namespace b200
