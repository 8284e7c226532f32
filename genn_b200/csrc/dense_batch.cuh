// DENSE delivery of a batched network: every weight row that a step needs is read once for all the copies that need it.
//
// The rows are what bounds it.  With 32 copies at 2.5 % a step reaches 55 % of the rows, 1.44 copies each; one pass over the
// rows per copy (presynapticPostSpanKernel) moves 1.44 times the bytes, and its threads wait for one load after another.
// Here a CTA owns DENSE_COLS columns and a range of source neurons.  It turns the copies' spike lists into one bit mask per
// source neuron (bit b: copy b spiked), gathers the sources that have one into a list, and its warps walk the list,
// DENSE_ROWS rows in flight each (12 warps x 8 x 512 bytes on an SM: what HBM's latency wants in flight).  A row's quad of
// columns is added to the private sums [copy][column] that every warp keeps in shared memory, where a lane only meets its
// own columns: plain loads and stores, no atomics.  The warps' sums are combined before one reduction per cell leaves the
// CTA, 16 bytes wide where the row allows.
//
// 8192 x 8192, 32 copies, 25 Hz at 1 ms (149 MB of rows a step): 107 us with presynapticPostSpanKernel, 55 here.
#pragma once

#include "common.cuh"
#include "presynaptic_update.cuh"

namespace b200
{
constexpr unsigned int DENSE_WARPS = 4;
constexpr unsigned int DENSE_BLOCK = DENSE_WARPS * 32;
constexpr unsigned int DENSE_COLS = 128;            // columns of a CTA: four a lane
constexpr unsigned int DENSE_COPIES = 32;           // copies of a CTA: one mask word
constexpr unsigned int DENSE_ROWS = 8;              // rows a warp has in flight
constexpr unsigned int DENSE_WINDOW = 2048;         // most source neurons of a CTA (masks and list: 12 KB)
// A CTA reads all spike lists to find its own sources: worth it while those are a small part of what it reads of the rows.
constexpr unsigned int DENSE_MOST_SOURCES = 65536;

struct DenseLaunch
{
    SynapseLaunch S;                    // DENSE groups that do not learn
    const uint4 *parts;                 // per CTA: group, first column, first source, number of sources
};

inline size_t denseSmemBytes(unsigned int copies, unsigned int window)
{
    return (size_t)DENSE_WARPS * copies * DENSE_COLS * sizeof(float) + window * (sizeof(unsigned int) + sizeof(uint16_t)) + 16u;
}

// Four columns of a row: a 16-byte load where rows keep that alignment, else four coalesced words.  (Lanes beyond the row's
// end read its last columns again; what they add is never flushed.)
template<bool VEC>
__device__ __forceinline__ float4 denseLoad(const float *row, unsigned int lane, unsigned int cols)
{
    if(VEC) return __ldg(reinterpret_cast<const float4*>(row + min(lane * 4u, cols - 4u)));
    return make_float4(__ldg(row + min(lane, cols - 1u)), __ldg(row + min(lane + 32u, cols - 1u)),
                       __ldg(row + min(lane + 64u, cols - 1u)), __ldg(row + min(lane + 96u, cols - 1u)));
}

// A lane's four sums of one copy (its columns as in denseLoad).
template<bool VEC>
__device__ __forceinline__ void denseAdd(float *sums, unsigned int lane, const float4 &w)
{
    if(VEC) {
        float4 *const at = reinterpret_cast<float4*>(sums) + lane;
        float4 a = *at;
        a.x = B200_FADD(a.x, w.x); a.y = B200_FADD(a.y, w.y); a.z = B200_FADD(a.z, w.z); a.w = B200_FADD(a.w, w.w);
        *at = a;
    }
    else {
        sums[lane] = B200_FADD(sums[lane], w.x);
        sums[lane + 32u] = B200_FADD(sums[lane + 32u], w.y);
        sums[lane + 64u] = B200_FADD(sums[lane + 64u], w.z);
        sums[lane + 96u] = B200_FADD(sums[lane + 96u], w.w);
    }
}

template<bool VEC>
__device__ __forceinline__ void denseRows(const b200_synapse_group &g, float *sums, const unsigned int *mask, const uint16_t *list,
                                          unsigned int listed, unsigned int firstColumn, unsigned int firstSource, unsigned int cols,
                                          unsigned int warp, unsigned int lane)
{
    const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    const float c = g.wu_params[0];
    const float *const base = constant ? nullptr : g.g + (unsigned long long)firstSource * g.num_trg + firstColumn;
    const unsigned int rowStride = g.num_trg;
    // the next rows are on their way while these are added; behind the list's end its last row is read again and not added
    auto fetch = [&](float4 (&w)[DENSE_ROWS], unsigned int (&m)[DENSE_ROWS], unsigned int first) {
        unsigned int s[DENSE_ROWS];
        #pragma unroll
        for(unsigned int j = 0; j < DENSE_ROWS; j++) s[j] = list[min(first + j, listed - 1u)];
        #pragma unroll
        for(unsigned int j = 0; j < DENSE_ROWS; j++) {
            w[j] = constant ? make_float4(c, c, c, c) : denseLoad<VEC>(base + (unsigned long long)s[j] * rowStride, lane, cols);
        }
        #pragma unroll
        for(unsigned int j = 0; j < DENSE_ROWS; j++) m[j] = (first + j < listed) ? mask[s[j]] : 0u;
    };
    auto add = [&](const float4 (&w)[DENSE_ROWS], const unsigned int (&m)[DENSE_ROWS]) {
        #pragma unroll
        for(unsigned int j = 0; j < DENSE_ROWS; j++) {
            for(unsigned int left = m[j]; left; left &= left - 1u) denseAdd<VEC>(sums + (unsigned int)(__ffs(left) - 1) * DENSE_COLS, lane, w[j]);
        }
    };
    constexpr unsigned int STRIDE = DENSE_WARPS * DENSE_ROWS;
    float4 wa[DENSE_ROWS], wb[DENSE_ROWS];
    unsigned int ma[DENSE_ROWS], mb[DENSE_ROWS];
    unsigned int first = warp * DENSE_ROWS;
    if(first >= listed) return;
    fetch(wa, ma, first);
    while(true) {
        if(first + STRIDE < listed) fetch(wb, mb, first + STRIDE);
        add(wa, ma);
        first += STRIDE;
        if(first >= listed) break;
        if(first + STRIDE < listed) fetch(wa, ma, first + STRIDE);
        add(wb, mb);
        first += STRIDE;
        if(first >= listed) break;
    }
}

static __global__ void __launch_bounds__(DENSE_BLOCK)
denseBatchKernel(const DenseLaunch L)
{
    extern __shared__ __align__(16) unsigned char denseShared[];
    __shared__ unsigned int listed;
    __shared__ unsigned int counts[DENSE_COPIES];
    const uint4 part = __ldg(&L.parts[blockIdx.x]);
    const b200_synapse_group &g = L.S.groups[part.x];
    const unsigned int firstCopy = blockIdx.z * DENSE_COPIES, copies = min(DENSE_COPIES, L.S.batch - firstCopy);
    chainWait();
    const unsigned int k = chainPhase(L.S.state, L.S.ahead);
    const unsigned int slots = g.src_delay_slots, slot = ringSlot(k + slots - g.axonal_delay, slots);
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned int cols = min(DENSE_COLS, g.num_trg - part.y);
    float *const sums = reinterpret_cast<float*>(denseShared);
    unsigned int *const mask = reinterpret_cast<unsigned int*>(sums + DENSE_WARPS * copies * DENSE_COLS);
    uint16_t *const list = reinterpret_cast<uint16_t*>(mask + part.w);

    if(threadIdx.x < copies) counts[threadIdx.x] = min(g.src_spk_cnt[(firstCopy + threadIdx.x) * slots + slot], g.num_src);
    if(threadIdx.x == 0u) listed = 0u;
    for(unsigned int i = threadIdx.x; i < part.w; i += DENSE_BLOCK) mask[i] = 0u;
    for(unsigned int i = threadIdx.x; i < DENSE_WARPS * copies * DENSE_COLS / 4u; i += DENSE_BLOCK) {
        reinterpret_cast<float4*>(sums)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    // ---- spike lists -> masks of this CTA's sources: a warp takes every DENSE_WARPS-th copy
    for(unsigned int b = warp; b < copies; b += DENSE_WARPS) {
        const unsigned int *const spk = g.src_spk + ((unsigned long long)(firstCopy + b) * slots + slot) * g.num_src;
        const unsigned int n = counts[b];
        for(unsigned int at = lane; at < n; at += 32u * 8u) {
            unsigned int id[8];
            #pragma unroll
            for(unsigned int j = 0; j < 8u; j++) id[j] = (at + 32u * j < n) ? spk[at + 32u * j] : 0xFFFFFFFFu;
            #pragma unroll
            for(unsigned int j = 0; j < 8u; j++) {
                if(id[j] - part.z < part.w) atomicOr(&mask[id[j] - part.z], 1u << b);
            }
        }
        if(L.S.count_events && lane == 0u && part.y == 0u && part.z == 0u) {
            atomicAdd(&L.S.state->synaptic_events, (unsigned long long)n * g.num_trg);
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
    const bool vec = (g.num_trg & 3u) == 0u;
    float *const own = sums + warp * copies * DENSE_COLS;
    if(vec) denseRows<true>(g, own, mask, list, rows, part.y, part.z, cols, warp, lane);
    else denseRows<false>(g, own, mask, list, rows, part.y, part.z, cols, warp, lane);
    __syncthreads();
    // ---- the warps' sums together, out to the targets' input
    const unsigned int quads = copies * DENSE_COLS / 4u;
    for(unsigned int q = threadIdx.x; q < quads; q += DENSE_BLOCK) {
        float4 a = reinterpret_cast<const float4*>(sums)[q];
        #pragma unroll
        for(unsigned int o = 1; o < DENSE_WARPS; o++) {
            const float4 x = reinterpret_cast<const float4*>(sums)[o * quads + q];
            a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
        }
        const unsigned int b = q / (DENSE_COLS / 4u), col = (q % (DENSE_COLS / 4u)) * 4u;
        if(col >= cols || (a.x == 0.0f && a.y == 0.0f && a.z == 0.0f && a.w == 0.0f)) continue;
        float *const out = g.out_post + (unsigned long long)(firstCopy + b) * g.num_trg + part.y + col;
        if(vec) {
            redAdd4(out, a);
        }
        else {
            redAdd(out, a.x);
            if(col + 1u < cols) redAdd(out + 1, a.y);
            if(col + 2u < cols) redAdd(out + 2, a.z);
            if(col + 3u < cols) redAdd(out + 3, a.w);
        }
    }
}
}   // namespace b200
