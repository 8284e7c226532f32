// SPARSE delivery of a batched network whose target buffers fit an SM's shared memory.
//
// One reduction into L2 per synaptic event is bound by the 1.9e11 scattered reductions a second that the L2 takes (measured;
// 8 M events: 42 us), one addition in shared memory by 8e11 (random cells
// of 4 MB and of 80 KB, all SMs, nothing else: 193 and 803 G a second).  A CTA takes one copy of one target buffer (outPost, or a whole
// dendritic-delay ring) into its shared memory as private sums, a share of that copy's spikes, and adds their rows as they
// lie in the model's arrays: whole rows, 6 to 9 bytes a synapse, no second copy of the synapses and no table of runs.  The
// sums go to the target once at the end, 16 bytes a reduction.  A share with few events (SCATTER_FEW) leaves the sums alone
// and reduces straight into L2: clearing and flushing them would take longer.
//
// Shares: the spikes of all groups onto the buffer stand on one line, each as long as its group's rows; a CTA owns an equal
// stretch of the line and computes it from the spike counts itself.  Inside, a warp takes pieces of SCATTER_PIECE synapses.
// They come as bulk copies into a ring of the warp's own (SCATTER_WARPS warps x 2 to 4 pieces of 1.5 to 2.3 KB: 50 KB and
// more under way on an SM, what HBM's latency wants, and no warp waits for another).  Pieces held in registers instead, one
// ahead: 27 KB under way and 37 instructions an event besides its addition, 43 us at the size below.
//
// 20 000 + 20 000 neurons, 8 copies, 8 M events a step: 90 us with the tiled kernels, 31 here (shared-memory pipe 53 %, issue slots 36 %).
#pragma once

#include <type_traits>

#include "common.cuh"
#include "presynaptic_update.cuh"

namespace b200
{
constexpr unsigned int SCATTER_BLOCK = 768;
constexpr unsigned int SCATTER_WARPS = SCATTER_BLOCK / 32;
constexpr unsigned int SCATTER_PIECE = 256;                             // synapses: eight a lane
constexpr unsigned int SCATTER_ALIGN = 16;                              // synapses: pieces start where every array allows a bulk copy
constexpr unsigned int SCATTER_MOST_DEPTH = 4;                          // pieces in a warp's ring
constexpr unsigned int SCATTER_SMEM = 225 * 1024;
constexpr unsigned int SCATTER_MOST_SOURCES = 64;                       // groups onto one buffer
constexpr unsigned int SCATTER_STAGED = 2;                              // of these in shared memory (with the rest of it, all an SM has)
// An event costs 0.19 ns of an SM's shared memory and 0.78 ns of its share of the L2's reductions; clearing and flushing
// the sums about 2.5 us.
constexpr unsigned int SCATTER_FEW = 4096;
// Spikes of a copy and step from which the kernel is used.  presynapticSparseKernel takes sixteen spikes of a copy side by side
// and the next sixteen behind them; this one starts its rings, clears and flushes whatever there is to do.  A step takes, with
// it / here: 1000 neurons, p = 0.1, 8 copies, 5 spikes a copy 5.9 / 7.8 us, 50 spikes 8.0 / 8.4; 3000 neurons, 15 spikes
// 6.6 / 7.8, 150 spikes 20.4 / 12.0; 10 000 neurons, 50 spikes 14.5 / 11.6 (p = 0.02: 10.0 / 9.3, with 32 copies 13.7 / 15.8).
constexpr float SCATTER_MIN_SPIKES = 64.0f;

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
    unsigned int cells;                 // of the largest buffer
    unsigned int depth;                 // pieces in a warp's ring
    unsigned int piece_bytes;
};

__device__ __forceinline__ void scatterShared(float *cell, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;" :: "r"((unsigned int)__cvta_generic_to_shared(cell)), "f"(v) : "memory");
}

__device__ __forceinline__ unsigned int scatterShare(const void *p) { return (unsigned int)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void scatterBulk(unsigned int to, const void *from, unsigned int bytes, unsigned int bar)
{
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(to), "l"(__cvta_generic_to_global(from)), "r"(bytes), "r"(bar) : "memory");
}

// A warp's ring of pieces.
struct ScatterRing
{
    unsigned char *data;
    unsigned long long *bars;
    unsigned int depth, bytes;          // pieces, bytes of one
    unsigned int sent, taken;           // slots of the next piece sent and taken
    unsigned int parity;                // of the slot next taken
    unsigned int polls;                 // for a piece before the step is given up
    bool failed;                        // it has been
};

// A lane's item: one piece of a spike's row.
struct ScatterItem
{
    unsigned long long first;           // synapse in the group's arrays
    unsigned int low, end;              // the row's synapses in the piece
};

// Four indices of a piece.
template<int IND>
__device__ __forceinline__ void scatterIndices(const unsigned char *data, unsigned int at, unsigned int (&cell)[4])
{
    if(IND == 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(data + at * 4u);
        cell[0] = v.x; cell[1] = v.y; cell[2] = v.z; cell[3] = v.w;
    }
    else if(IND == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(data + at * 2u);
        cell[0] = v.x & 0xFFFFu; cell[1] = v.x >> 16; cell[2] = v.y & 0xFFFFu; cell[3] = v.y >> 16;
    }
    else {
        const unsigned int v = *reinterpret_cast<const unsigned int*>(data + at);
        cell[0] = v & 0xFFu; cell[1] = (v >> 8) & 0xFFu; cell[2] = (v >> 16) & 0xFFu; cell[3] = v >> 24;
    }
}

// A wait ran out: the pieces on their way have to arrive before the block ends.  (Out of line: six instances of its caller wait for
// instructions as it is.)
static __device__ __noinline__ void scatterGiveUp(StepState *state, const unsigned long long *bars, unsigned int depth, unsigned int slot,
                                                  unsigned int parity, unsigned int sent)
{
    atomicOr(&state->error, ERR_COPY_TIMEOUT);
    for(; sent; sent--) {
        copyArrived(bars + slot, parity, COPY_WAITS);
        if(++slot == depth) {
            slot = 0;
            parity ^= 1u;
        }
    }
}

// What a warp does of one group's spikes: pieces `item`, `item` + SCATTER_WARPS, ... of the group's; returns how far beyond
// them its next one lies.  The widths are template parameters: they decide every address.
template<int IND, bool DELAYS>
__device__ __forceinline__ unsigned int scatterGroup(const SynapseLaunch &S, const b200_synapse_group &g, const unsigned int *spk, unsigned int spikes,
                                                     unsigned int item, ScatterRing &R, float *sums, float *cells, bool few, unsigned int front)
{
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int stride = g.row_stride, numTrg = g.num_trg, D = g.max_den_delay, numSrc = g.num_src;
    const unsigned int pieces = (stride + SCATTER_ALIGN - 1u + SCATTER_PIECE - 1u) / SCATTER_PIECE, items = spikes * pieces;
    const unsigned int n = items > item ? (items - item + SCATTER_WARPS - 1u) / SCATTER_WARPS : 0u;
    const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    const float c = g.wu_params[0];
    // a lane looks up one of 32 consecutive items
    auto look = [&](unsigned int from) {
        ScatterItem I{0ull, 0u, 0u};
        const unsigned int turn = from + lane;
        if(turn < n) {
            const unsigned int x = item + turn * SCATTER_WARPS, spike = x / pieces, offset = (x - spike * pieces) * SCATTER_PIECE;
            const unsigned int pre = spk[spike];
            if(pre < numSrc) {
                const unsigned int length = __ldg(&g.row_length[pre]);
                const unsigned long long rowStart = (unsigned long long)pre * stride;
                const unsigned int skew = (unsigned int)rowStart & (SCATTER_ALIGN - 1u);
                I.first = rowStart - skew + offset;
                I.low = skew > offset ? skew - offset : 0u;
                I.end = skew + length > offset ? min(skew + length - offset, SCATTER_PIECE) : 0u;
                if(S.count_events && offset == 0u) atomicAdd(&S.state->synaptic_events, (unsigned long long)length);
            }
            else atomicOr(&S.state->error, ERR_IND_RANGE);
        }
        return I;
    };
    auto send = [&](const ScatterItem &I) {
        // (whole groups of SCATTER_ALIGN: behind the arrays' last row that is in their padding)
        const unsigned int m = (I.end + SCATTER_ALIGN - 1u) & ~(SCATTER_ALIGN - 1u);
        const unsigned int bar = scatterShare(R.bars + R.sent), to = scatterShare(R.data + R.sent * R.bytes);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(m * (IND + (constant ? 0u : 4u) + (DELAYS ? 1u : 0u))) : "memory");
        if(m) {
            scatterBulk(to, static_cast<const unsigned char*>(g.ind) + I.first * IND, m * IND, bar);
            if(!constant) scatterBulk(to + SCATTER_PIECE * IND, g.g + I.first, m * 4u, bar);
            if(DELAYS) scatterBulk(to + SCATTER_PIECE * (IND + 4u), g.d + I.first, m, bar);
        }
    };
    auto next = [&](unsigned int &slot) { slot = (slot + 1u == R.depth) ? 0u : slot + 1u; };
    auto add = [&](const unsigned char *data, unsigned int low, unsigned int end) {
        #pragma unroll
        for(unsigned int q = 0; q < SCATTER_PIECE / 128u; q++) {
            const unsigned int at = q * 128u + lane * 4u;
            if(at >= end) break;
            unsigned int cell[4];
            scatterIndices<IND>(data, at, cell);
            const float4 v = constant ? make_float4(c, c, c, c) : *reinterpret_cast<const float4*>(data + SCATTER_PIECE * IND + at * 4u);
            const float w[4] = {v.x, v.y, v.z, v.w};
            const unsigned int delay = DELAYS ? *reinterpret_cast<const unsigned int*>(data + SCATTER_PIECE * (IND + 4u) + at) : 0u;
            auto place = [&](unsigned int j) {
                if(DELAYS) {
                    unsigned int slot = front + ((delay >> (8u * j)) & 0xFFu);
                    while(slot >= D) slot -= D;         // a delay of the ring length or more wraps around
                    cell[j] += slot * numTrg;
                }
            };
            // the quads inside a row, all but its first and last, need no test of their own for every synapse
            if(at >= low && at + 4u <= end && max(max(cell[0], cell[1]), max(cell[2], cell[3])) < numTrg) {
                #pragma unroll
                for(unsigned int j = 0; j < 4u; j++) place(j);
                if(few) {
                    #pragma unroll
                    for(unsigned int j = 0; j < 4u; j++) redAdd(cells + cell[j], w[j]);
                }
                else {
                    #pragma unroll
                    for(unsigned int j = 0; j < 4u; j++) scatterShared(sums + cell[j], w[j]);
                }
            }
            else {
                #pragma unroll
                for(unsigned int j = 0; j < 4u; j++) {
                    if(at + j < low || at + j >= end) continue;
                    if(cell[j] >= numTrg) {
                        atomicOr(&S.state->error, ERR_IND_RANGE);
                        continue;
                    }
                    place(j);
                    if(few) redAdd(cells + cell[j], w[j]);
                    else scatterShared(sums + cell[j], w[j]);
                }
            }
        }
    };
    ScatterItem here = look(0u), later = {0ull, 0u, 0u};
    for(unsigned int turn = 0; turn < min(n, R.depth); turn++) {
        if(lane == turn) send(here);
        next(R.sent);
    }
    for(unsigned int turn = 0; turn < n; turn++) {
        const unsigned int at = turn & 31u;
        if(at == 0u) {
            if(turn) here = later;
            later = look(turn + 32u);
        }
        const unsigned int low = __shfl_sync(0xFFFFFFFFu, here.low, at), end = __shfl_sync(0xFFFFFFFFu, here.end, at);
        const bool there = copyArrived(R.bars + R.taken, R.parity, R.polls);
        if(there) add(R.data + R.taken * R.bytes, low, end);
        // the lanes' vote after the piece, not before it: each waits for itself
        if(!__all_sync(0xFFFFFFFFu, there)) {
            scatterGiveUp(S.state, R.bars, R.depth, R.taken, R.parity, min(n, turn + R.depth) - turn);
            R.failed = true;
            break;
        }
        __syncwarp();
        next(R.taken);
        if(R.taken == 0u) R.parity ^= 1u;
        if(turn + R.depth < n) {
            const unsigned int ahead = (turn + R.depth) & 31u;
            if(lane == ahead) send(ahead < at ? later : here);
            next(R.sent);
        }
    }
    return item + n * SCATTER_WARPS - items;
}

static __global__ void __launch_bounds__(SCATTER_BLOCK, 1)
sparseBatchKernel(const ScatterLaunch L)
{
    extern __shared__ __align__(16) float scatterSums[];
    __shared__ __align__(8) unsigned long long scatterBars[SCATTER_WARPS][SCATTER_MOST_DEPTH];
    __shared__ unsigned int firstSpike[SCATTER_MOST_SOURCES], spikes[SCATTER_MOST_SOURCES];
    unsigned long long *const line = reinterpret_cast<unsigned long long*>(scatterSums + ((L.cells + 31u) & ~31u));     // (until pieces come into the rings)
    const ScatterPart part = L.parts[blockIdx.x];
    const ScatterTarget T = L.targets[part.target];
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    // (common.cuh: stageGroup; the groups of a buffer, where they are few)
    __shared__ __align__(16) b200_synapse_group stagedGroups[SCATTER_STAGED];
    const bool staged = T.num_groups <= SCATTER_STAGED;
    if(staged) stageWords(stagedGroups, L.S.groups + T.first_group, sizeof(b200_synapse_group) * T.num_groups);
    const b200_synapse_group *const groups = staged ? stagedGroups : L.S.groups + T.first_group;
    if(lane < L.depth) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(scatterShare(&scatterBars[warp][lane])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // (the sums are cleared while the kernel before this one ends, whether they will be needed or not)
    for(unsigned int i = threadIdx.x; i < (T.num_cells + 3u) / 4u; i += SCATTER_BLOCK) {
        reinterpret_cast<float4*>(scatterSums)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    chainWait();
    const unsigned int k = chainPhase(L.S.state, L.S.ahead), polls = L.S.state->copy_wait_limit;
    // ---- this CTA's stretch of the line of spikes
    if(threadIdx.x < T.num_groups) {
        const b200_synapse_group &g = groups[threadIdx.x];
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
        const unsigned int stride = max(1u, groups[threadIdx.x].row_stride);
        auto from = [&](unsigned long long at) {
            return at <= before ? 0u : (unsigned int)min((unsigned long long)spikes[threadIdx.x], (at - before + stride - 1u) / stride);
        };
        const unsigned int first = from(low);
        firstSpike[threadIdx.x] = first;
        spikes[threadIdx.x] = from(high) - first;
    }
    // (`line` lies where bulk copies are about to write)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    float *const cells = T.cells + (unsigned long long)part.copy * T.num_cells;
    ScatterRing ring{reinterpret_cast<unsigned char*>(scatterSums + ((L.cells + 31u) & ~31u)) + (size_t)warp * L.depth * L.piece_bytes,
                     scatterBars[warp], L.depth, L.piece_bytes, 0u, 0u, 0u, polls, false};
    unsigned int item = warp;
    for(unsigned int gi = 0; gi < T.num_groups && !ring.failed; gi++) {
        const b200_synapse_group &g = groups[gi];
        const unsigned int slots = g.src_delay_slots, slot = ringSlot(k + slots - g.axonal_delay, slots);
        const unsigned int *const spk = g.src_spk + ((unsigned long long)part.copy * slots + slot) * g.num_src + firstSpike[gi];
        const unsigned int front = g.max_den_delay ? ringSlot(k + 1u, g.max_den_delay) : 0u;
        auto deliver = [&](auto ind, auto delays) {
            item = scatterGroup<decltype(ind)::value, decltype(delays)::value>(L.S, g, spk, spikes[gi], item, ring, scatterSums, cells, few, front);
        };
        using std::integral_constant;
        if(g.max_den_delay) {
            if(g.ind_bytes == 2u) deliver(integral_constant<int, 2>(), integral_constant<bool, true>());
            else if(g.ind_bytes == 4u) deliver(integral_constant<int, 4>(), integral_constant<bool, true>());
            else deliver(integral_constant<int, 1>(), integral_constant<bool, true>());
        }
        else if(g.ind_bytes == 2u) deliver(integral_constant<int, 2>(), integral_constant<bool, false>());
        else if(g.ind_bytes == 4u) deliver(integral_constant<int, 4>(), integral_constant<bool, false>());
        else deliver(integral_constant<int, 1>(), integral_constant<bool, false>());
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
