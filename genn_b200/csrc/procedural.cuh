// PROCEDURAL fixed-probability connectivity with drawn weights: rows regenerated for every spike.
//
// Instructions bound it: a Philox block for four gaps, another for every weight, two logarithms, a root and a cosine per
// synapse, and the L2 takes 1.9e11 scattered reductions a second.  With one thread per sub-row from its first draw to its
// last delivery a warp took as long as its longest sub-row (21 of 32 lanes busy), eight warp instructions an event.  Here a
// warp works in two phases.  Its lanes regenerate the targets of the sub-rows of one or more spikes (a gap needs a quarter of
// the instructions of a synapse), then all targets are moved together, row by row, and the lanes share the rows' weights
// and deliveries evenly.  A lane that overruns its PROC_HOLD targets keeps its place and goes on when the held ones
// are delivered.  The logarithm's quotient and the root are one rounding of the exact result each, as in
// genn_b200_rng.h, without the branches of the general division and root; Philox's round keys come as launch parameters.
//
// 1 M neurons, 1000 synapses each, 32 sub-rows, a step of 1.2e9 events: 11.5 ms before, 7.1 here (the reductions alone: 6.4).
#pragma once

#include "common.cuh"
#include "init.cuh"
#include "presynaptic_update.cuh"

namespace b200
{
constexpr unsigned int DRAWN_BLOCK = 128;
constexpr unsigned int PROC_WARPS = DRAWN_BLOCK / 32;
constexpr unsigned int PROC_HOLD = 48;              // targets of a lane between the phases
constexpr unsigned int PROC_LANE = PROC_HOLD + 1;   // odd: lanes at the same place of their targets meet no bank conflict
constexpr unsigned int PROC_PER_SM = 8;
// A lane may take several neighbouring sub-rows of a spike: when they are short (below, `PROC_FILL` targets expected), the
// four draws of their last Philox blocks and the rounds of the slowest lane would be most of the work.
constexpr float PROC_FILL = 24.0f;

struct ProceduralKeys { unsigned int k[20]; };      // Philox's keys, round after round

inline ProceduralKeys proceduralKeys(unsigned long long seed)
{
    ProceduralKeys K;
    unsigned int k0 = (unsigned int)seed, k1 = (unsigned int)(seed >> 32);
    for(int r = 0; r < 10; r++) {
        K.k[2 * r] = k0;
        K.k[2 * r + 1] = k1;
        k0 += B200_PHILOX_W0;
        k1 += B200_PHILOX_W1;
    }
    return K;
}

struct ProceduralLaunch
{
    SynapseLaunch S;
    ProceduralKeys keys;
};

__device__ __forceinline__ uint4 proceduralPhilox(const ProceduralKeys &K, unsigned int c0, unsigned int c1, unsigned int c2, unsigned int c3)
{
    #pragma unroll
    for(int r = 0; r < 10; r++) {
        const unsigned long long p0 = (unsigned long long)B200_PHILOX_M0 * c0, p1 = (unsigned long long)B200_PHILOX_M1 * c2;
        c0 = (unsigned int)(p1 >> 32) ^ c1 ^ K.k[2 * r];
        c1 = (unsigned int)p1;
        c2 = (unsigned int)(p0 >> 32) ^ c3 ^ K.k[2 * r + 1];
        c3 = (unsigned int)p0;
    }
    return make_uint4(c0, c1, c2, c3);
}

// b200_u32_to_uniform: (k + 1/2) 2^-23 from 1 + k 2^-23, both exact.
__device__ __forceinline__ float proceduralUniform(unsigned int x)
{
    return B200_FADD(__uint_as_float((x >> 9) | 0x3F800000u), -0.999999940395355224609375f);
}

// b200_logf for the uniforms, equal for every one of the 2^23 (tests/test_procedural_math.py, as are the others here).  The quotient of numbers in [-0.3, 0.42]
// and [1.7, 2.42] needs no scaling: an approximate reciprocal, and the quotient corrected by its exact remainder (Markstein,
// IBM J. Res. Dev. 34, 1990).
__device__ __forceinline__ float proceduralLog(float u)
{
    const unsigned int bits = __float_as_uint(u);
    const int a = (int)(bits - 0x3F3504F4u);            // sqrt(1/2): the mantissas of [sqrt(1/2), sqrt(2))
    const float m = __uint_as_float(bits - ((unsigned int)a & 0xFF800000u));
    const float e = B200_FADD(__uint_as_float(0x4B400000u + (unsigned int)(a >> 23)), -12582912.0f);
    const float n = B200_FSUB(m, 1.0f), d = B200_FADD(m, 1.0f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = B200_FMUL(n, r);
    const float s = B200_FMAF(B200_FMAF(-d, q, n), r, q);
    const float s2 = B200_FMUL(s, s);
    float p = 0.2222222222f;
    p = B200_FMAF(p, s2, 0.2857142857f);
    p = B200_FMAF(p, s2, 0.4f);
    p = B200_FMAF(p, s2, 0.6666666667f);
    p = B200_FMAF(p, s2, 2.0f);
    return B200_FMAF(e, 0.6931471805599453f, B200_FMUL(p, s));
}

// Root of a number far from the ends of the range, corrected by its exact remainder (the same reference).
__device__ __forceinline__ float proceduralRoot(float y)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    const float g = B200_FMUL(y, r);
    return B200_FMAF(B200_FMAF(-g, g, y), B200_FMUL(0.5f, r), g);
}

// The cosine of b200_sincos2pif for a uniform: 4 u rounded is its nearest quarter turn (no uniform lies between two).
__device__ __forceinline__ float proceduralCos(float u)
{
    const float z = B200_FMAF(u, 4.0f, 12582912.0f);
    const unsigned int q = __float_as_uint(z);
    const float r = B200_FMUL(B200_FMAF(B200_FADD(z, -12582912.0f), -0.25f, u), 6.283185307179586f);
    const float r2 = B200_FMUL(r, r);
    float sp = B200_FMAF(-1.9841269841e-04f, r2, 8.3333333333e-03f);
    sp = B200_FMAF(sp, r2, -1.6666666667e-01f);
    sp = B200_FMAF(B200_FMUL(sp, r2), r, r);
    float cp = B200_FMAF(2.4801587302e-05f, r2, -1.3888888889e-03f);
    cp = B200_FMAF(cp, r2, 4.1666666667e-02f);
    cp = B200_FMAF(cp, r2, -0.5f);
    cp = B200_FMAF(cp, r2, 1.0f);
    // quarter turns 0..3: cos, -sin, -cos, sin
    return __uint_as_float(__float_as_uint((q & 1u) ? sp : cp) ^ (((q + 1u) & 2u) << 30));
}

// The weight of one element of its stream.  (WIDE: element numbers of more than 32 bits)
template<bool NORMAL, bool WIDE>
__device__ __forceinline__ float proceduralWeight(const ProceduralKeys &K, const b200_synapse_group &g, unsigned long long seed,
                                                  unsigned int stream, unsigned long long element, float mean, float sd)
{
    if(NORMAL) {
        const uint4 x = proceduralPhilox(K, (unsigned int)element, stream, WIDE ? (unsigned int)(element >> 32) : 0u, 0x80000000u);
        const float rad = proceduralRoot(B200_FMUL(-2.0f, proceduralLog(proceduralUniform(x.x))));
        return B200_FADD(mean, B200_FMUL(B200_FMUL(rad, proceduralCos(proceduralUniform(x.y))), sd));
    }
    b200_rng rng = b200_rng_init(seed, stream, element);
    return drawInitValue(g.proc_weight_init, g.proc_weight_params, &rng);
}

// Where a lane stands in its sub-rows.
struct ProceduralPlace
{
    unsigned int sub;                   // sub-row
    unsigned int block;                 // next Philox block of its stream
    int last;                           // last target, counted from the sub-row's first
};

template<bool NORMAL, bool WIDE>
static __global__ void __launch_bounds__(DRAWN_BLOCK, PROC_PER_SM)
proceduralDrawnKernel(const ProceduralLaunch L)
{
    __shared__ unsigned int heldAll[PROC_WARPS][32 * PROC_LANE];
    __shared__ unsigned int slotEnds[PROC_WARPS][32];
    __shared__ unsigned long long slotElements[PROC_WARPS][32];
    const b200_synapse_group &g = L.S.groups[blockIdx.y];
    const unsigned int b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const bool noAutapse = (g.proc_connect == B200_CONNECT_FIXED_PROBABILITY_NO_AUTAPSE);
    const unsigned int T = connectSubRows(g.proc_connect, g.proc_connect_params);
    const unsigned int numTrg = g.num_trg, numSrc = g.num_src, stride = g.row_stride;
    const unsigned int per = (numTrg + T - 1u) / T;
    const float recip = g.proc_connect_params[1];
    const unsigned int stream = g.rng_stream, weightStream = g.proc_weight_stream;
    const float mean = g.proc_weight_params[0], sd = g.proc_weight_params[1];
    unsigned int *const held = heldAll[warp];
    unsigned int *const slotEnd = slotEnds[warp];
    unsigned long long *const slotElement = slotElements[warp];
    chainWait();
    const unsigned int k = chainPhase(L.S.state, L.S.ahead);
    const unsigned int slots = g.src_delay_slots, rslot = ringSlot(k + slots - g.axonal_delay, slots);
    const unsigned int count = min(g.src_spk_cnt[b * slots + rslot], numSrc);
    const unsigned int *const spk = g.src_spk + ((unsigned long long)b * slots + rslot) * numSrc;
    const unsigned int D = g.max_den_delay;
    // dendritic delay is not generated procedurally: slot 0 of a ring is the front
    float *const target = (D ? g.den_delay + ((unsigned long long)b * D + ringSlot(k + 1, D)) * numTrg : g.out_post + (unsigned long long)b * numTrg);
    const unsigned int warps = gridDim.x * PROC_WARPS;
    // lanes of a spike: fewer while their targets still fit and every warp still has a spike
    unsigned int G = T;
    while(G > 1u && g.proc_connect_params[0] * (float)per * (float)(T / G) * 2.0f <= PROC_FILL && (unsigned long long)count * (G / 2u) >= 32ull * warps) G >>= 1;
    const unsigned int R = T / G, S = 32u / G;
    const unsigned int slot = lane / G, first = (lane % G) * R;
    auto deliver = [&](unsigned long long element, unsigned int post) {
        redAdd(target + post, proceduralWeight<NORMAL, WIDE>(L.keys, g, L.S.seed, weightStream, element, mean, sd));
    };
    for(unsigned int base = (blockIdx.x * PROC_WARPS + warp) * S; base < count; base += warps * S) {
        unsigned int pre = 0;
        bool more = base + slot < count;
        if(more) {
            pre = spk[base + slot];
            if(pre >= numSrc) {
                atomicOr(&L.S.state->error, ERR_IND_RANGE);
                more = false;
            }
        }
        const bool live = more;
        const unsigned long long rowElement = (unsigned long long)pre * stride;
        ProceduralPlace at{first, 0u, -1}, resume = at;
        unsigned int n = 0, kept = 0;
        // ---- targets: one Philox block, four gaps a round
        auto rounds = [&](bool counting) {
            // (a lane that runs out of room goes on counting the first time, and stops after that)
            const bool asked = more;
            bool room = more;
            unsigned int m = 0;
            kept = 0;
            while(__any_sync(0xFFFFFFFFu, more)) {
                if(!more) continue;
                if(room && m + 4u > PROC_HOLD) {
                    room = false;
                    resume = at;
                    if(!counting) {
                        more = false;
                        continue;
                    }
                }
                const unsigned int low = at.sub * per;
                if(low >= numTrg) {
                    more = false;
                    continue;
                }
                const unsigned int span = min(per, numTrg - low);
                const unsigned long long element = (unsigned long long)pre * T + at.sub;
                const uint4 x = proceduralPhilox(L.keys, (unsigned int)element, stream, (unsigned int)(element >> 32), 0x80000000u + at.block);
                const unsigned int word[4] = {x.x, x.y, x.z, x.w};
                bool inside = true;
                #pragma unroll
                for(int i = 0; i < 4; i++) {
                    const int j = at.last + 1 + (int)B200_FMUL(proceduralLog(proceduralUniform(word[i])), recip);
                    if(inside) at.last = j;
                    inside = inside && (unsigned int)j < span;
                    if(inside && !(noAutapse && (unsigned int)j + low == pre)) {
                        if(room) held[lane * PROC_LANE + m] = (unsigned int)j + low;
                        m++;
                    }
                }
                if(room) kept = m;
                if(inside) at.block++;
                else {
                    at = ProceduralPlace{at.sub + 1u, 0u, -1};
                    more = at.sub < first + R;
                }
            }
            if(counting) n = m;
            more = asked && !room;              // there is a rest to regenerate
            at = resume;
        };
        rounds(true);
        __syncwarp();
        // ---- a row's length; a lane's first synapse in its row
        unsigned int upTo = n;
        for(unsigned int o = 1; o < G; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, upTo, o);
            if(lane % G >= o) upTo += v;
        }
        const unsigned int length = __shfl_sync(0xFFFFFFFFu, upTo, slot * G + G - 1u);
        const bool tooLong = live && length > stride;
        if(live && lane % G == 0u) {
            if(tooLong) atomicOr(&L.S.state->error, ERR_IND_RANGE);
            if(L.S.count_events) atomicAdd(&L.S.state->synaptic_events, (unsigned long long)min(length, stride));
        }
        if(!__any_sync(0xFFFFFFFFu, more || tooLong)) {
            // ---- all targets together, lane after lane: a lane's only move towards the front
            unsigned int end = n;
            #pragma unroll
            for(unsigned int o = 1; o < 32u; o <<= 1) {
                const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, end, o);
                if(lane >= o) end += v;
            }
            const unsigned int total = __shfl_sync(0xFFFFFFFFu, end, 31);
            for(unsigned int from = 1; from < 32u; from++) {
                const unsigned int m = __shfl_sync(0xFFFFFFFFu, n, from), to = __shfl_sync(0xFFFFFFFFu, end, from) - m;
                const unsigned int *const own = held + from * PROC_LANE;
                const unsigned int v0 = lane < m ? own[lane] : 0u, v1 = lane + 32u < m ? own[lane + 32u] : 0u;
                __syncwarp();
                if(lane < m) held[to + lane] = v0;
                if(lane + 32u < m) held[to + lane + 32u] = v1;
                __syncwarp();
            }
            if(lane % G == G - 1u) {
                slotEnd[slot] = end;
                slotElement[slot] = rowElement - (end - length);
            }
            __syncwarp();
            // ---- weights and deliveries, shared evenly
            unsigned int row = 0, rowEnd = slotEnd[0];
            unsigned long long element = slotElement[0];
            for(unsigned int i = lane; i < total; i += 32u) {
                while(i >= rowEnd) {
                    row++;
                    rowEnd = slotEnd[row];
                    element = slotElement[row];
                }
                deliver(element + i, held[i]);
            }
            __syncwarp();
        }
        else {
            // ---- a lane has more than it can hold, or a row more than its stride: lane after lane, the held targets, then the rest
            unsigned int done = upTo - n;       // place in the row of the first one held
            while(true) {
                for(unsigned int from = 0; from < 32u; from++) {
                    const unsigned int m = __shfl_sync(0xFFFFFFFFu, kept, from), place = __shfl_sync(0xFFFFFFFFu, done, from);
                    const unsigned long long element = __shfl_sync(0xFFFFFFFFu, rowElement, from);
                    for(unsigned int i = lane; i < m; i += 32u) {
                        if(place + i < stride) deliver(element + place + i, held[from * PROC_LANE + i]);
                    }
                }
                done += kept;
                __syncwarp();
                if(!__any_sync(0xFFFFFFFFu, more)) break;
                kept = 0;
                rounds(false);
                __syncwarp();
            }
        }
    }
}
}   // namespace b200
