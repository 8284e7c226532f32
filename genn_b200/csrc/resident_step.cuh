// Time steps of the target-resident kernel: see resident.h.  Its instances are compiled in four units (resident_*.cu).
#pragma once

#include "resident.h"
#include "common.cuh"

namespace b200
{
__device__ __forceinline__ unsigned long long loadRelaxedGpu(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ ulonglong2 loadRelaxedGpu(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void storeRelaxedGpu(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void storeRelaxedGpu(ulonglong2 *p, unsigned long long x, unsigned long long y)
{
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" :: "l"(p), "l"(x), "l"(y) : "memory");
}

// Bytes on their way into L2 (both multiples of 16).
__device__ __forceinline__ void prefetchL2(const void *p, unsigned int bytes)
{
    if(bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ void residentAdd(float *cell, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;" :: "r"((unsigned int)__cvta_generic_to_shared(cell)), "f"(v) : "memory");
}

// ---- time steps ----------------------------------------------------------------------------------
// The commonest neurons (LIF, one or two exponential inputs, at most one Poisson source; spike sources) without neuronCompute's
// choices of a model: its operations in its order, constants side by side in shared memory, places of the inputs in registers.
// An SM with 21 warps of neurons is bound by their instructions, a smaller one by the chain of them: with the choices, a neuron
// of two conductances took 1100 cycles of a step, one of a current input 500.
struct ResidentLif
{
    float vthresh, vreset, vrest, ioffset;
    float rmembrane, exp_tc, tau_refrac, cs_init;
    float cs_decay, pad[3];
    struct { float level, decay; } input[2];    // EXP_CURR: its factor, EXP_COND: its reversal potential
};

// What a warp's neurons are (bits).
constexpr unsigned int RESIDENT_IS_LIF = 1u, RESIDENT_IS_POISSON = 2u, RESIDENT_IS_ARRAY = 4u, RESIDENT_IS_DRAWN = 8u, RESIDENT_IS_SOURCE = 16u,
                       RESIDENT_HAS_INPUT = 32u, RESIDENT_HAS_TWO = 64u, RESIDENT_COND = 128u, RESIDENT_COND_TWO = 256u;

struct ResidentShared
{
    unsigned int depth[RESIDENT_CLASSES], columns[RESIDENT_CLASSES], base[RESIDENT_CLASSES];
    // (three of each, in turn: warps are at most one barrier apart, and a step may have only one)
    unsigned int list[3][RESIDENT_LIST];        // neuron group << 24 | neuron
    unsigned int listed[3];                     // spikes in the list (counts on beyond its end)
    unsigned int stop[3];                       // 1: a wait ran out, 2: this launch has lost enough, 4: more spikes than the list holds
    unsigned int sent[2];                       // this CTA's spikes of the step, and how many
    __align__(16) unsigned short ids[2][RESIDENT_BLOCK];
    unsigned int firstWarp[RESIDENT_MAX_GROUPS + 1];    // warps of this CTA before those of each group
    unsigned long long done;                    // StepState at the start of the launch
    unsigned int phase, period;
    unsigned int limit;                         // polls of a wait
    int debt;                                   // ns lost, by thread 0's account up to the step `accounted`
    unsigned int accounted;
    unsigned int steps;                         // of this launch (every thread writes a smaller number for itself when it ends early)
    __align__(16) ResidentLif lif[RESIDENT_MAX_GROUPS];
};

// Front buffers of the ring classes, in registers of every thread (all threads advance them alike).
template<bool ONE>
struct ResidentFronts
{
    unsigned int f[RESIDENT_CLASSES];
    __device__ __forceinline__ unsigned int operator[](unsigned int c) const { return (c == 0u) ? f[0] : (c == 1u) ? f[1] : (c == 2u) ? f[2] : f[3]; }
};

// One ring class: where its front buffer begins, the columns of a buffer, and all of them.
template<>
struct ResidentFronts<true>
{
    unsigned int at, columns, all;
    __device__ __forceinline__ void advance() { at = (at + columns == all) ? 0u : at + columns; }
    __device__ __forceinline__ void back() { at = (at == 0u) ? all - columns : at - columns; }
};

extern __shared__ __align__(16) unsigned char residentSmem[];

// Thread 0's account of a step with more than a few spikes (resident.h: "Busy networks"); the steps since the last such one made
// up for half of `spare` each at least.  (Nothing is done in the others: every instruction is on the chain of the step.)
__device__ __forceinline__ void residentAccount(ResidentShared &sh, unsigned int weight, unsigned int spare, unsigned int patience, unsigned int step,
                                             unsigned int spikes, unsigned int *stop)
{
    int debt = sh.debt;
    if(sh.accounted <= step) {
        debt = max(debt - (int)(min(step - sh.accounted, 1u << 14) * (spare / 2u)), 0) - (int)spare;
        sh.accounted = step + 1u;
    }
    debt = min(debt + (int)(min(spikes, RESIDENT_LIST) * weight) + (spikes > RESIDENT_LIST ? (int)RESIDENT_PIECE_COST : 0), (int)RESIDENT_MOST_DEBT);
    sh.debt = debt;
    if(debt > 0 && (unsigned int)debt > patience) atomicOr(stop, 2u);
}

template<typename T>
__device__ __forceinline__ T *residentTable(unsigned int at)
{
    return reinterpret_cast<T*>(residentSmem + at);
}

// What a warp has in flight of one item of the runs.
struct ResidentHeld
{
    uint2 e[RESIDENT_LOADS];
};

// Spikes of a list onto this CTA's neurons.  ONE: a model with one ring class and one axonal delay.
template<bool ONE>
struct ResidentDeliver
{
    using Fronts = ResidentFronts<ONE>;
    const ResidentLaunch &L;
    const ResidentShared &sh;
    unsigned int events;

    __device__ __forceinline__ unsigned int warp() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ unsigned int warps() const { return blockDim.x >> 5; }
    __device__ __forceinline__ unsigned int lane() const { return threadIdx.x & 31u; }

    __device__ __forceinline__ void add(unsigned int cls, unsigned int delay, unsigned int col, float v, const Fronts &front)
    {
        float *const acc = residentTable<float>(L.at.acc);
        if constexpr(ONE) {
            unsigned int at = front.at + delay * front.columns;
            if(at >= front.all) at -= front.all;
            residentAdd(acc + at + col, v);
        }
        else {
            unsigned int slot = front[cls] + delay;
            const unsigned int D = sh.depth[cls];
            if(slot >= D) slot -= D;
            residentAdd(acc + sh.base[cls] + slot * sh.columns[cls] + col, v);
        }
        events++;
    }

    // loads of item `it` of the runs: a spike, or a share of one whose run is long (every `chunks`-th group of 32 entries, so that
    // the padding behind the longest run is shared out too: as stretches, the last of them was little but padding)
    __device__ __forceinline__ void fetch(ResidentHeld &H, const unsigned int *list, unsigned int a, unsigned int n, unsigned int it) const
    {
        #pragma unroll
        for(unsigned int u = 0; u < RESIDENT_LOADS; u++) H.e[u] = make_uint2(RESIDENT_PAD, 0u);
        const unsigned int chunks = L.chunks[a];
        if(it >= n * chunks) return;
        const unsigned int s = (chunks == 1u) ? it : it / chunks;
        const unsigned int spike = list[s];
        const ResidentRun run = (residentTable<const ResidentRun>(L.at.runs) + a * L.neuron.num_groups)[spike >> 24];
        const unsigned int i = (it - s * chunks) * 32u + lane(), step = 32u * chunks;
        const uint2 *p = L.entries + run.base() + run.near() + (unsigned long long)(spike & 0xFFFFFFu) * run.row + i;
        #pragma unroll
        for(unsigned int u = 0; u < RESIDENT_LOADS; u++) if(i + u * step < run.length) H.e[u] = __ldg(p + u * step);
    }

    __device__ __forceinline__ void addHeld(const ResidentHeld &H, const Fronts &front)
    {
        #pragma unroll
        for(unsigned int u = 0; u < RESIDENT_LOADS; u++) {
            const uint2 e = H.e[u];
            if(e.x != RESIDENT_PAD) add(e.x >> 30, (e.x >> 16) & 0x3FFFu, e.x & 0xFFFFu, __uint_as_float(e.y), front);
        }
    }

    // items of the runs from `it` on, two at a time
    __device__ __forceinline__ void runs(const unsigned int *list, unsigned int a, unsigned int n, unsigned int it, const Fronts &front)
    {
        for(const unsigned int items = n * L.chunks[a]; it < items; it += 2u * warps()) {
            ResidentHeld H, H2;
            fetch(H, list, a, n, it);
            fetch(H2, list, a, n, it + warps());
            addHeld(H, front);
            addHeld(H2, front);
        }
    }

    // heads of the runs: all of the list's spikes as one line of entries
    __device__ __forceinline__ void near(const unsigned int *list, unsigned int a, unsigned int n, const Fronts &front)
    {
        const unsigned int most = L.near_most[a], share = L.near_share[a], items = n * most;
        for(unsigned int it = threadIdx.x; it < items; it += RESIDENT_NEAR_LOADS * blockDim.x) {
            uint2 e[RESIDENT_NEAR_LOADS];
            #pragma unroll
            for(unsigned int u = 0; u < RESIDENT_NEAR_LOADS; u++) {
                const unsigned int item = it + u * blockDim.x;
                e[u] = make_uint2(RESIDENT_PAD, 0u);
                if(item >= items) continue;
                // (items: at most 2048 spikes of 64 entries, so the product's upper half is the quotient)
                const unsigned int s = (most == 1u) ? item : __umulhi(item, share), i = item - s * most;
                const unsigned int spike = list[s];
                const ResidentRun run = (residentTable<const ResidentRun>(L.at.runs) + a * L.neuron.num_groups)[spike >> 24];
                if(i < run.near()) e[u] = __ldg(L.entries + run.base() + (unsigned long long)(spike & 0xFFFFFFu) * run.row + i);
            }
            #pragma unroll
            for(unsigned int u = 0; u < RESIDENT_NEAR_LOADS; u++) {
                if(e[u].x != RESIDENT_PAD) add(e[u].x >> 30, 0u, e[u].x & 0xFFFFu, __uint_as_float(e[u].y), front);
            }
        }
    }

    // DENSE and BITMASK groups, into the buffer `ahead` steps ahead
    __device__ __forceinline__ void spans(const unsigned int *list, unsigned int a, unsigned int n, unsigned int ahead, const Fronts &front)
    {
        for(unsigned int q = 0; q < L.num_spans; q++) {
            const ResidentSpan &S = residentTable<const ResidentSpan>(L.at.spans)[q];
            if(S.delay_class != a) continue;
            const unsigned int w0 = sh.firstWarp[S.trg_group], targets = sh.firstWarp[S.trg_group + 1] - w0;
            if(!targets) continue;
            const unsigned int *gp = S.gp, src = S.src_group, numTrg = S.num_trg;
            const unsigned int per = gp ? 32u : RESIDENT_DENSE_SPIKES;
            const unsigned int items = targets * ((n + per - 1u) / per);
            for(unsigned int it = warp(); it < items; it += warps()) {
                const unsigned int part = (targets == 1u) ? it : it / targets, w = w0 + (it - part * targets);
                // this unit's place in its population: 32 targets, one word of a BITMASK row
                const unsigned int unit = w * gridDim.x + blockIdx.x - residentTable<const unsigned int>(L.at.unit_start)[S.trg_group];
                const unsigned int post = unit * 32u + lane();
                const unsigned int from = part * per;
                float sum = 0.0f;
                if(gp) {
                    unsigned int word = 0;
                    const unsigned int spike = (from + lane() < n) ? list[from + lane()] : 0xFFFFFFFFu;
                    if((spike >> 24) == src) word = __ldg(&gp[(((unsigned long long)(spike & 0xFFFFFFu) * S.row_stride) >> 5) + unit]);
                    // bit 31 - lane of the words of all lanes
                    unsigned int c = 0;
                    #pragma unroll
                    for(unsigned int b = 0; b < 32u; b++) {
                        const unsigned int who = __ballot_sync(0xFFFFFFFFu, (word >> (31u - b)) & 1u);
                        if(lane() == b) c = who;
                    }
                    if(post < numTrg) {
                        events += __popc(c);
                        sum = (float)__popc(c) * S.weight;
                    }
                }
                else {
                    // (ids first, then all loads, then the sum: nothing waits in between)
                    const float *g = S.g;
                    float w8[RESIDENT_DENSE_SPIKES];
                    #pragma unroll
                    for(unsigned int u = 0; u < RESIDENT_DENSE_SPIKES; u++) {
                        const unsigned int spike = (from + u < n) ? list[from + u] : 0xFFFFFFFFu;
                        const bool take = (spike >> 24) == src && post < numTrg;
                        w8[u] = (take && !g) ? S.weight : 0.0f;
                        if(take && g) w8[u] = __ldg(&g[(unsigned long long)(spike & 0xFFFFFFu) * numTrg + post]);
                        events += take ? 1u : 0u;
                    }
                    #pragma unroll
                    for(unsigned int u = 0; u < RESIDENT_DENSE_SPIKES; u++) sum += w8[u];
                }
                const unsigned int col = residentTable<const unsigned int>(L.at.columns)[w * B200_MAX_PSM + S.psm];
                if(sum != 0.0f) {
                    add(col >> 16, ahead, (col & 0xFFFFu) + lane(), sum, front);
                    events--;           // (counted above)
                }
            }
        }
    }
};

// The Poisson draws of a neuron's one current source: a Philox block holds four time steps, and a step computes a share of
// the ten rounds of the next block instead of all of them.
struct ResidentDraws
{
    b200_philox_out now, next;

    __device__ __forceinline__ void start(unsigned long long seed, unsigned int stream, unsigned int element, unsigned long long timestep)
    {
        now = b200_rng_step_block(seed, stream, element, timestep);
        // the rounds of the next block that earlier steps would have done
        const unsigned int j = (unsigned int)timestep & 3u;
        begin(stream, element, timestep);
        if(j > 0u) rounds<0, 3>(seed);
        if(j > 1u) rounds<3, 6>(seed);
        if(j > 2u) rounds<6, 8>(seed);
    }
    __device__ __forceinline__ void begin(unsigned int stream, unsigned int element, unsigned long long timestep)
    {
        const unsigned long long blk = (timestep >> 2) + 1ull;
        next.x[0] = element; next.x[1] = stream; next.x[2] = (unsigned int)blk; next.x[3] = ((unsigned int)(blk >> 32) & 0x7FFFu) << 16;
    }
    template<int FROM, int TO>
    __device__ __forceinline__ void rounds(unsigned long long seed)
    {
        #pragma unroll
        for(int r = FROM; r < TO; r++) {
            const unsigned long long p0 = (unsigned long long)B200_PHILOX_M0 * next.x[0], p1 = (unsigned long long)B200_PHILOX_M1 * next.x[2];
            const unsigned int n0 = (unsigned int)(p1 >> 32) ^ next.x[1] ^ ((unsigned int)seed + (unsigned int)r * B200_PHILOX_W0);
            const unsigned int n2 = (unsigned int)(p0 >> 32) ^ next.x[3] ^ ((unsigned int)(seed >> 32) + (unsigned int)r * B200_PHILOX_W1);
            next.x[1] = (unsigned int)p1;
            next.x[3] = (unsigned int)p0;
            next.x[0] = n0;
            next.x[2] = n2;
        }
    }
    // the uniform of this time step
    __device__ __forceinline__ float draw(unsigned long long seed, unsigned int stream, unsigned int element, unsigned long long timestep)
    {
        const float u = b200_u32_to_uniform(b200_rng_step_word(&now, timestep));
        switch((unsigned int)timestep & 3u) {
        case 0: rounds<0, 3>(seed); break;
        case 1: rounds<3, 6>(seed); break;
        case 2: rounds<6, 8>(seed); break;
        default:
            rounds<8, 10>(seed);
            now = next;
            begin(stream, element, timestep + 1ull);
        }
        return u;
    }
};

// b200_poisson_inverse from the cumulative probabilities it would add up (the host made them with the same operations).
__device__ __forceinline__ unsigned int residentPoisson(float u, const float *table)
{
    unsigned int n = 0;
    for(; n < 64u; n += 4u) {
        const float4 s = *reinterpret_cast<const float4*>(table + n);
        const unsigned int c = (u > s.x ? 1u : 0u) + (u > s.y ? 1u : 0u) + (u > s.z ? 1u : 0u) + (u > s.w ? 1u : 0u);
        if(c < 4u) return n + c;
    }
    return n;
}

__device__ __forceinline__ void residentLifTable(ResidentLif &q, const b200_neuron_group &g)
{
    q.vthresh = g.params[0]; q.vreset = g.params[1]; q.vrest = g.params[2]; q.ioffset = g.params[3];
    q.rmembrane = g.params[4]; q.exp_tc = g.params[5]; q.tau_refrac = g.params[6];
    q.cs_init = g.cs[0].params[0]; q.cs_decay = g.cs[0].params[1];
    for(int i = 0; i < 2; i++) {
        const bool cond = g.psm[i].model == B200_PSM_EXP_COND;
        q.input[i].level = g.psm[i].params[cond ? 1 : 0];
        q.input[i].decay = g.psm[i].params[cond ? 0 : 1];
    }
}

// `table`: Poisson sources have their counts looked up (residentPoisson).
template<int NCS>
__device__ __forceinline__ unsigned int residentWhat(const b200_neuron_group &g, bool source, bool table)
{
    unsigned int what = source ? RESIDENT_IS_SOURCE : 0u;
    const bool drawn = NCS == 1 && table && g.num_cs && g.cs[0].model == B200_CS_POISSON_EXP;
    if(drawn) what |= RESIDENT_IS_DRAWN;
    bool plain = g.num_psm <= 2u && (g.num_cs == 0u || drawn);
    for(unsigned int p = 0; p < min(g.num_psm, 2u); p++) plain = plain && (g.psm[p].model == B200_PSM_EXP_CURR || g.psm[p].model == B200_PSM_EXP_COND);
    if(g.model == B200_NEURON_LIF && plain) {
        what |= RESIDENT_IS_LIF;
        if(g.num_psm > 0u) what |= RESIDENT_HAS_INPUT | (g.psm[0].model == B200_PSM_EXP_COND ? RESIDENT_COND : 0u);
        if(g.num_psm > 1u) what |= RESIDENT_HAS_TWO | (g.psm[1].model == B200_PSM_EXP_COND ? RESIDENT_COND_TWO : 0u);
    }
    if(g.num_psm == 0u && g.num_cs == 0u) {
        if(g.model == B200_NEURON_POISSON) what |= RESIDENT_IS_POISSON;
        if(g.model == B200_NEURON_SPIKE_SOURCE_ARRAY) what |= RESIDENT_IS_ARRAY;
    }
    return what;
}

// What a launch leaves behind of its account: `debt` at its end, `done` steps by then.
__device__ __forceinline__ void residentSettle(const ResidentLaunch &L, StepState &state, int debt, unsigned int step, unsigned long long done)
{
    if(step < L.num_steps || (unsigned int)debt > L.patience) {
        const unsigned int rest = min(max(2u * state.resident_rest, RESIDENT_REST), RESIDENT_MOST_REST);
        state.resident_rest = rest;
        state.resident_hold = done + rest;
        state.resident_debt = min((unsigned int)debt, L.patience - L.patience / 4u);       // (the next time it is seen sooner)
        *reinterpret_cast<volatile unsigned long long*>(L.hold) = done + rest;
    }
    else {
        // (as many steps without that make up for one time)
        state.resident_rest -= min(state.resident_rest, step);
        state.resident_debt = (unsigned int)debt;
    }
}

template<int NPSM, int NCS>
__device__ __forceinline__ bool residentLif(const ResidentLif &q, float dt, NeuronRegs<NPSM, NCS> &r, const float (&in)[NPSM], unsigned int what, unsigned int count)
{
    float V = __uint_as_float(r.v[0]), R = __uint_as_float(r.v[1]), Isyn = 0.0f;
    #pragma unroll
    for(unsigned int p = 0; p < (NPSM < 2 ? NPSM : 2); p++) {
        if(what & (p ? RESIDENT_HAS_TWO : RESIDENT_HAS_INPUT)) {
            const float lin = B200_FADD(r.lin[p], in[p]), level = q.input[p].level;
            const float factor = (what & (p ? RESIDENT_COND_TWO : RESIDENT_COND)) ? B200_FSUB(level, V) : level;
            Isyn = B200_FADD(Isyn, B200_FMUL(lin, factor));
            r.lin[p] = B200_FMUL(lin, q.input[p].decay);
        }
    }
    if(NCS > 0 && (what & RESIDENT_IS_DRAWN)) {
        const float current = B200_FADD(r.cs[0], B200_FMUL(q.cs_init, (float)count));
        Isyn = B200_FADD(Isyn, current);
        r.cs[0] = B200_FMUL(current, q.cs_decay);
    }
    const float alpha = B200_FADD(B200_FMUL(B200_FADD(Isyn, q.ioffset), q.rmembrane), q.vrest);
    const float moved = B200_FSUB(alpha, B200_FMUL(q.exp_tc, B200_FSUB(alpha, V)));
    const bool free = R <= 0.0f;
    V = free ? moved : V;
    R = free ? R : B200_FSUB(R, dt);
    const bool spiked = R <= 0.0f && V >= q.vthresh;
    r.v[0] = __float_as_uint(spiked ? q.vreset : V);
    r.v[1] = __float_as_uint(spiked ? q.tau_refrac : R);
    return spiked;
}

// BLOCK: most threads.  With 640 a thread has 96 registers and next to nothing is spilled, with 768 it has 80.
template<int NPSM, int NCS, bool ONE, unsigned int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1)
residentStepKernel(const __grid_constant__ ResidentLaunch L)
{
    __shared__ ResidentShared sh;
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const unsigned int numGroups = L.neuron.num_groups;
    const unsigned int G = gridDim.x, me = blockIdx.x;
    const unsigned int numDelays = ONE ? 1u : L.num_delays;
    const b200_neuron_group *const groups = residentTable<const b200_neuron_group>(L.at.groups);
    const unsigned int *const unitFirst = residentTable<const unsigned int>(L.at.unit_first);
    float *const acc = residentTable<float>(L.at.acc);
    // tables into shared memory
    stageWordsAsync(residentSmem + L.at.groups, L.neuron.groups, sizeof(b200_neuron_group) * numGroups);
    stageWordsAsync(residentSmem + L.at.unit_start, L.unit_start, sizeof(unsigned int) * (numGroups + 1));
    stageWordsAsync(residentSmem + L.at.unit_first, L.unit_first, sizeof(unsigned int) * L.num_units);
    stageWordsAsync(residentSmem + L.at.columns, L.columns + (size_t)me * RESIDENT_UNITS * B200_MAX_PSM, sizeof(unsigned int) * RESIDENT_UNITS * B200_MAX_PSM);
    stageWordsAsync(residentSmem + L.at.runs, L.runs + (size_t)me * numDelays * numGroups, sizeof(ResidentRun) * numDelays * numGroups);
    stageWordsAsync(residentSmem + L.at.rows, L.rows, sizeof(unsigned long long) * numDelays * numGroups);
    stageWordsAsync(residentSmem + L.at.spans, L.spans, sizeof(ResidentSpan) * L.num_spans);
    if(L.poisson) stageWordsAsync(residentSmem + L.at.poisson, L.poisson, sizeof(float) * 64u * numGroups);
    StepState *const state = L.neuron.state;
    const unsigned long long t0 = state->timestep;
    if(L.may_leave) {
        if(me == 0 && threadIdx.x == 0) *L.barrier = 0ull;
        if(state->steps_done < state->resident_hold) {              // (the same for every CTA: both change at the end of a launch)
            stagedWords();
            return;
        }
    }
    if(threadIdx.x == 0) {
        sh.debt = (int)state->resident_debt;
        sh.accounted = 0u;
        sh.steps = L.num_steps;
        unsigned int base = 0;
        for(unsigned int c = 0; c < RESIDENT_CLASSES; c++) {
            const unsigned int n = (c < L.num_depths) ? L.cta_columns[me * RESIDENT_CLASSES + c] : 0u;
            sh.depth[c] = (c < L.num_depths) ? L.depth[c] : 1u;
            sh.columns[c] = n;
            sh.base[c] = base;
            base += n * sh.depth[c];
        }
        for(int i = 0; i < 3; i++) sh.listed[i] = sh.stop[i] = 0u;
        sh.sent[0] = sh.sent[1] = 0u;
        sh.done = state->steps_done;
        sh.phase = state->phase;
        sh.period = state->ring_period;
        sh.limit = (unsigned int)min(state->barrier_spin_limit, 0xFFFFFFFFull);
    }
    for(unsigned int i = threadIdx.x; i < L.acc_floats; i += blockDim.x) acc[i] = 0.0f;
    for(unsigned int i = threadIdx.x; i < numGroups; i += blockDim.x) residentLifTable(sh.lif[i], L.neuron.groups[i]);
    stagedWords();
    __syncthreads();
    const unsigned int no0 = (unsigned int)sh.done;         // (step numbers of messages: 20 bits)
    // (up to 65 entries; the option "resident_warps" allows blocks of 32 threads)
    for(unsigned int i = threadIdx.x; i <= numGroups; i += blockDim.x) {
        // first warp whose unit (warp * G + me) is not before the group
        const unsigned int u = residentTable<const unsigned int>(L.at.unit_start)[i];
        sh.firstWarp[i] = (u <= me) ? 0u : (u - me + G - 1u) / G;
    }
    ResidentFronts<ONE> front;
    if constexpr(ONE) {
        front.columns = sh.columns[0];
        front.all = sh.depth[0] * front.columns;
        front.at = ((sh.phase + 1u) % sh.depth[0]) * front.columns;
    }
    else {
        #pragma unroll
        for(unsigned int c = 0; c < RESIDENT_CLASSES; c++) front.f[c] = (sh.phase + 1u) % sh.depth[c];
    }

    // this thread's neuron
    const bool mine = warp < RESIDENT_UNITS && warp * G + me < L.num_units;
    unsigned int group = 0, local = 0;
    bool active = false;
    unsigned int what = 0;          // RESIDENT_IS_... (the same for a whole warp)
    float nextTime = 0.0f;          // RESIDENT_IS_ARRAY: of the next spike
    NeuronRegs<NPSM, NCS> regs;
    unsigned int myCol[NPSM];       // ring class << 24 | place of buffer 0 of this neuron's input
    ResidentDraws draws;
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) myCol[p] = 0u;
    if(mine) {
        group = unitFirst[warp * G + me] >> 24;
        local = (unitFirst[warp * G + me] & 0xFFFFFFu) + lane;
        const b200_neuron_group &g = groups[group];
        active = local < g.num_update;
        what = residentWhat<NCS>(g, (L.source_groups >> group) & 1ull, L.poisson != nullptr);
        #pragma unroll
        for(unsigned int p = 0; p < NPSM; p++) {
            const unsigned int col = residentTable<const unsigned int>(L.at.columns)[warp * B200_MAX_PSM + p], c = col >> 16;
            myCol[p] = (c << 24) | (sh.base[c] + (col & 0xFFFFu) + lane);
        }
        if(active) {
            loadNeuron<true>(g, local, regs);
            #pragma unroll
            for(unsigned int p = 0; p < NPSM; p++) {
                if(p < g.num_psm && g.psm[p].max_den_delay) {
                    const unsigned int c = myCol[p] >> 24, n = sh.columns[c];
                    float *cell = acc + (myCol[p] & 0xFFFFFFu);
                    const float *ring = g.psm[p].den_delay + local;
                    #pragma unroll 8
                    for(unsigned int d = 0; d < sh.depth[c]; d++) cell[d * n] = __ldcg(ring + (size_t)d * g.num_neurons);
                }
            }
            if(what & RESIDENT_IS_DRAWN) draws.start(L.neuron.seed, g.cs[0].rng_stream, local, t0);
            if((what & RESIDENT_IS_ARRAY) && regs.v[0] != regs.v[1]) nextTime = __ldg(&g.egp[regs.v[0]]);
        }
    }
    ResidentDeliver<ONE> deliver{L, sh, 0u};
    unsigned int buf = (unsigned int)((sh.done + 1ull) % L.buffers);      // buffer of the message of this step
    unsigned int recAt = L.neuron.num_recording_timesteps ? (unsigned int)(t0 % L.neuron.num_recording_timesteps) : 0u;
    unsigned int histAt = 0, turn = 0, spikes = 0;
    // the last warps ask for the messages, one sender per lane; the very last one sends this CTA's own
    const unsigned int asked = (warps - 1u - warp) * 32u + lane;
    const unsigned int myCell = (me % L.copies) * G + asked;
    auto gaveUp = [&](unsigned int &polls, unsigned int *stop) -> bool {
        if(++polls <= sh.limit) return false;
        atomicOr(&state->error, ERR_BARRIER_TIMEOUT);
        atomicOr(stop, 1u);
        return true;
    };
    // the sender's cell of the step with number `no` (bounded wait); the second word only if it is needed
    auto awaitCell = [&](unsigned int from, unsigned int no, unsigned int *stop) -> ulonglong2 {
        const ulonglong2 *p = L.inbox + (from * L.copies * G + myCell);
        const unsigned int tag = no << 12;      // as it stands in the upper half of a word
        unsigned int polls = 0;
        for(;;) {
            const ulonglong2 w = loadRelaxedGpu(p);
            const unsigned int hi = (unsigned int)(w.x >> 32) ^ tag;
            if(hi < 4096u && ((hi >> 2) <= RESIDENT_HEAD_IDS || ((unsigned int)(w.y >> 32) ^ tag) < 4096u)) return w;
            if(gaveUp(polls, stop)) return make_ulonglong2(0ull, 0ull);
        }
    };
    // spike `i` of a message
    auto spikeOf = [&](const ulonglong2 &w, unsigned int i, unsigned int from, unsigned int no, unsigned int *stop) -> unsigned int {
        unsigned int id;
        if(i < RESIDENT_HEAD_IDS) id = (unsigned int)(w.x >> (10u * i));
        else if(i < RESIDENT_CELL_IDS) id = (unsigned int)(w.y >> (10u * (i - RESIDENT_HEAD_IDS)));
        else {
            const unsigned int j = (i - RESIDENT_CELL_IDS) / RESIDENT_MORE_IDS;
            const unsigned long long *p = L.more + ((size_t)from * G + asked) * L.more_words + j;
            unsigned long long v;
            unsigned int polls = 0;
            while((unsigned int)((v = loadRelaxedGpu(p)) >> 44) != (no & (unsigned int)(RESIDENT_TAG_STEPS - 1ull))) {
                if(gaveUp(polls, stop)) { v = 0; break; }
            }
            id = (unsigned int)(v >> (10u * ((i - RESIDENT_CELL_IDS) % RESIDENT_MORE_IDS)));
        }
        id &= 0x3FFu;
        return unitFirst[min((id >> 5) * G + asked, L.num_units - 1u)] + (id & 31u);
    };
    __syncthreads();

    for(unsigned int step = 0; step < L.num_steps; step++) {
        // this step's random draws, while the messages are on their way
        unsigned int csCount[NCS > 0 ? NCS : 1] = {0};
        if(mine && active && !(what & RESIDENT_IS_ARRAY) && (NCS > 0 || !(what & RESIDENT_IS_LIF))) {
            const b200_neuron_group &g = groups[group];
            if(NCS == 1 && (what & RESIDENT_IS_DRAWN)) {
                csCount[0] = residentPoisson(draws.draw(L.neuron.seed, g.cs[0].rng_stream, local, t0 + step), residentTable<const float>(L.at.poisson) + 64u * group);
            }
            else drawCurrentSources<NCS>(L.neuron, g, 0u, local, t0 + step, csCount);
            if(g.model == B200_NEURON_POISSON) {
                residentTable<unsigned int>(L.at.undrawn)[threadIdx.x] = regs.v[0];
                if(__uint_as_float(regs.v[0]) <= 0.0f) {
                    regs.v[0] = __float_as_uint(drawPoissonInterval(L.neuron, g, 0u, local, t0 + step, __uint_as_float(regs.v[0])));
                }
            }
        }

        // ---------------- the spikes that reach their targets in this step (LATE: in the next) --------------------
        const unsigned int *heldList = nullptr;     // the last class's list, if some of its runs wait for the neuron update
        unsigned int heldCount = 0;
        for(unsigned int a = 0; a < numDelays; a++) {
            const unsigned int kind = L.kind[a], late = (kind == RESIDENT_LATE) ? 1u : 0u;
            if(step <= L.delay[a]) {
                // spikes from before this launch come from the spike lists, one piece after the other (a LATE class: in the
                // first step also those that are due in it)
                for(unsigned int ahead = (late && step == 0u) ? 0u : late; ahead <= late; ahead++) {
                    if(step + ahead >= L.delay[a] + 1u || (late && ahead && (step + 1u == L.num_steps || (numDelays > 1u && step + 1u == sh.steps)))) continue;
                    __syncthreads();
                    for(unsigned int gi = 0; gi < numGroups; gi++) {
                        if(!((L.sources[a] >> gi) & 1ull)) continue;
                        const b200_neuron_group &g = groups[gi];
                        const unsigned int slots = g.num_delay_slots, slot = ringSlot(sh.phase + step + ahead + slots - L.delay[a], slots);
                        const unsigned int n = min(__ldcg(&g.spk_cnt[slot]), g.num_neurons);
                        if(threadIdx.x == 0 && n > L.quiet[a]) residentAccount(sh, L.weight[a], L.spare, L.may_leave ? L.patience : ~0u, step, min(n, RESIDENT_LIST), &sh.stop[turn]);
                        for(unsigned int from = 0; from < n; from += RESIDENT_LIST) {
                            const unsigned int m = min(RESIDENT_LIST, n - from);
                            for(unsigned int i = threadIdx.x; i < m; i += blockDim.x) {
                                const unsigned int id = __ldcg(&g.spk[(size_t)slot * g.num_neurons + from + i]);
                                sh.list[turn][i] = (gi << 24) | min(id, g.num_neurons - 1u);
                                if(id >= g.num_neurons) atomicOr(&state->error, ERR_IND_RANGE);
                            }
                            __syncthreads();
                            // (entries of a LATE class say one step ahead)
                            ResidentFronts<ONE> at = front;
                            if(late && !ahead) {
                                if constexpr(ONE) at.back();
                                else {
                                    #pragma unroll
                                    for(unsigned int c = 0; c < RESIDENT_CLASSES; c++) at.f[c] = (at.f[c] == 0u) ? sh.depth[c] - 1u : at.f[c] - 1u;
                                }
                            }
                            if(kind == RESIDENT_SPLIT) deliver.near(sh.list[turn], a, m, at);
                            deliver.runs(sh.list[turn], a, m, warp, at);
                            deliver.spans(sh.list[turn], a, m, late, at);
                            __syncthreads();
                        }
                    }
                }
            }
            if(late && (step + 1u == L.num_steps || (numDelays > 1u && step + 1u == sh.steps))) {
                __syncthreads();            // (the next launch takes those; the update still waits for what the last step added)
                continue;
            }
            if(step + late <= L.delay[a]) continue;
            unsigned int had = 0, n = 0;
            ulonglong2 w = make_ulonglong2(0ull, 0ull);
            for(bool first = true;; first = false) {
                unsigned int *const list = sh.list[turn];
                if(asked < G) {
                    const unsigned int back = L.delay[a] + 1u - late, no = no0 + step + 1u - back;
                    const unsigned int from = (buf >= back) ? buf - back : buf + L.buffers - back;
                    if(first) {
                        w = awaitCell(from, no, &sh.stop[turn]);
                        n = (unsigned int)(w.x >> 34) & 0x3FFu;
                    }
                    if(n > had) {
                        if(ONE) {
                            unsigned int at = atomicAdd(&sh.listed[turn], n - had);
                            if(at + (n - had) > RESIDENT_LIST && first && L.may_leave) atomicOr(&sh.stop[turn], 4u);
                            for(; had < n && at < RESIDENT_LIST; had++, at++) list[at] = spikeOf(w, had, from, no, &sh.stop[turn]);
                        }
                        else {
                            // (spikes of groups without synapses of this delay take no room)
                            for(; had < n; had++) {
                                const unsigned int spike = spikeOf(w, had, from, no, &sh.stop[turn]);
                                if(!((L.sources[a] >> (spike >> 24)) & 1ull)) continue;
                                const unsigned int at = atomicAdd(&sh.listed[turn], 1u);
                                if(at >= RESIDENT_LIST) {
                                    if(first && L.may_leave && numDelays == 1u) atomicOr(&sh.stop[turn], 4u);
                                    break;
                                }
                                list[at] = spike;
                            }
                        }
                    }
                }
                __syncthreads();
                if(const unsigned int stop = sh.stop[turn]) {       // (written in front of the barrier only: the same for every thread)
                    if(stop & 1u) return;
                    if(first && a == 0u) {                          // 2 and 4: with `may_leave` only
                        if(numDelays > 1u || (BLOCK > RESIDENT_FEW && !late)) sh.steps = step + 1u;     // (this step is the last)
                        else if(late) {
                            // (the next step's spikes, which the next launch takes)
                            sh.steps = step + 1u;
                            break;
                        }
                        else if constexpr(BLOCK <= RESIDENT_FEW) {
                            // (this step is the other kernel's: drawn again, the same, with it.  The jump costs registers that
                            // the larger blocks do not have: +0.2 us a step)
                            if(mine && active && groups[group].model == B200_NEURON_POISSON) regs.v[0] = residentTable<unsigned int>(L.at.undrawn)[threadIdx.x];
                            sh.steps = step;
                            goto ended;
                        }
                    }
                }
                const unsigned int all = sh.listed[turn], m = min(all, RESIDENT_LIST);
                if(threadIdx.x == 0) {
                    sh.listed[turn == 0u ? 2u : turn - 1u] = 0u;
                    if(all > L.quiet[a]) residentAccount(sh, L.weight[a], L.spare, L.may_leave ? L.patience : ~0u, step, all, &sh.stop[turn == 2u ? 0u : turn + 1u]);
                }
                turn = (turn == 2u) ? 0u : turn + 1u;
                // (a LATE class in a step that has just become the last: for the next launch)
                if(m && !(numDelays > 1u && late && step + 1u == sh.steps)) {
                    // runs of the last class that may wait for the neuron update
                    if(kind != RESIDENT_IMMEDIATE && all <= RESIDENT_LIST && a + 1u == numDelays) {
                        heldList = list;
                        heldCount = m;
                        break;
                    }
                    if(kind == RESIDENT_SPLIT) deliver.near(list, a, m, front);
                    deliver.runs(list, a, m, warp, front);
                    deliver.spans(list, a, m, late, front);
                    // (nothing of a LATE class is for this step's update)
                    if(!late) __syncthreads();
                }
                if(all <= RESIDENT_LIST) break;
            }
        }
        // (loaded here and nowhere else, so that no copy between registers waits for the loads)
        ResidentHeld held;
        if(heldList) {
            const unsigned int a = numDelays - 1u;
            deliver.fetch(held, heldList, a, heldCount, warp);
            if(L.kind[a] == RESIDENT_SPLIT) {
                deliver.near(heldList, a, heldCount, front);
                __syncthreads();
            }
        }
        // ---------------- neuron update -------------------------------------------------------------------
        const unsigned int par = step & 1u;
        unsigned int ballot = 0;
        if(mine) {
            const b200_neuron_group &g = groups[group];
            bool spiked = false;
            if(active) {
                if(what & (RESIDENT_IS_POISSON | RESIDENT_IS_ARRAY)) {
                    if(what & RESIDENT_IS_POISSON) {
                        const float left = B200_FSUB(__uint_as_float(regs.v[0]), 1.0f);
                        spiked = left <= 0.0f;
                        regs.v[0] = __float_as_uint(left);
                    }
                    else if(regs.v[0] != regs.v[1] && B200_FMUL((float)(t0 + step), L.neuron.dt) >= nextTime) {
                        spiked = true;
                        if(++regs.v[0] != regs.v[1]) nextTime = __ldg(&g.egp[regs.v[0]]);
                    }
                }
                else {
                    float in[NPSM];
                    #pragma unroll
                    for(unsigned int p = 0; p < NPSM; p++) {
                        in[p] = 0.0f;
                        if((what & RESIDENT_IS_LIF) ? p < 2u && (what & (p ? RESIDENT_HAS_TWO : RESIDENT_HAS_INPUT)) : p < g.num_psm) {
                            float *cell = acc;
                            if constexpr(ONE) cell += myCol[p] + front.at;
                            else cell += (myCol[p] & 0xFFFFFFu) + front[myCol[p] >> 24] * sh.columns[myCol[p] >> 24];
                            const float v = *cell;
                            *cell = 0.0f;
                            if((what & RESIDENT_IS_LIF) || g.psm[p].max_den_delay) in[p] = v;
                            else regs.lin[p] = B200_FADD(regs.lin[p], v);
                        }
                    }
                    if(what & RESIDENT_IS_LIF) spiked = residentLif(sh.lif[group], L.neuron.dt, regs, in, what, csCount[0]);
                    else spiked = neuronCompute(L.neuron, g, 0u, local, t0 + step, B200_FMUL((float)(t0 + step), L.neuron.dt), regs, in, csCount, true);
                }
            }
            ballot = __ballot_sync(0xFFFFFFFFu, spiked);
            if(ballot && (what & RESIDENT_IS_SOURCE)) {
                unsigned int at = 0;
                if(lane == 0) at = atomicAdd(&sh.sent[par], __popc(ballot));
                at = __shfl_sync(0xFFFFFFFFu, at, 0);
                if(spiked) {
                    sh.ids[par][at + __popc(ballot & ((1u << lane) - 1u))] = (unsigned short)threadIdx.x;
                    // its rows, while the message is on its way (lengths are multiples of four entries)
                    if(L.prefetch) {
                        for(unsigned int a = 0; a < numDelays; a++) {
                            const unsigned int row = residentTable<const ResidentRun>(L.at.runs)[a * numGroups + group].row;
                            prefetchL2(L.entries + residentTable<const unsigned long long>(L.at.rows)[a * numGroups + group] + (size_t)local * row,
                                       row * (unsigned int)sizeof(uint2));
                        }
                    }
                }
            }
        }
        // ---------------- the message: sent by the last warp, waited for by no other ---------------------------
        if(warp == warps - 1u) {
            asm volatile("bar.sync 1, %0;" :: "r"(blockDim.x) : "memory");
            const unsigned long long tag = (unsigned long long)(no0 + step + 1u) << 44;
            const unsigned int total = sh.sent[par];
            unsigned long long w0 = tag, w1 = tag;
            if(total) {
                // (eight ids in one load; those beyond `total` are left from earlier steps and ignored by everybody)
                const uint4 v = *reinterpret_cast<const uint4*>(sh.ids[par]);
                w0 |= ((unsigned long long)total << 34) | (v.x & 0x3FFu) | ((v.x >> 16) & 0x3FFu) << 10 | (v.y & 0x3FFu) << 20;
                w1 |= ((v.y >> 16) & 0x3FFu) | (v.z & 0x3FFu) << 10 | ((v.z >> 16) & 0x3FFu) << 20 | (unsigned long long)(v.w & 0x3FFu) << 30;
            }
            if(lane < L.copies) storeRelaxedGpu(L.inbox + ((buf * L.copies + lane) * G + me), w0, w1);
            if(total > RESIDENT_CELL_IDS) {
                unsigned long long *more = L.more + ((size_t)buf * G + me) * L.more_words;
                for(unsigned int j = lane; j * RESIDENT_MORE_IDS + RESIDENT_CELL_IDS < total; j += 32u) {
                    unsigned long long w = tag;
                    for(unsigned int i = 0; i < RESIDENT_MORE_IDS; i++) {
                        const unsigned int at = RESIDENT_CELL_IDS + j * RESIDENT_MORE_IDS + i;
                        if(at < total) w |= (unsigned long long)sh.ids[par][at] << (10u * i);
                    }
                    storeRelaxedGpu(more + j, w);
                }
            }
            __syncwarp();
            if(lane == 0) sh.sent[par] = 0u;
        }
        else {
            asm volatile("bar.arrive 1, %0;" :: "r"(blockDim.x) : "memory");
        }
        if(mine && lane == 0) {
            residentTable<unsigned int>(L.at.history)[histAt * RESIDENT_UNITS + warp] = ballot;
            if(L.neuron.num_recording_timesteps && groups[group].record_spk) {
                groups[group].record_spk[(size_t)recAt * ((groups[group].num_update + 31u) / 32u) + local / 32u] = ballot;
            }
            spikes += __popc(ballot);
        }
        // ---------------- what had to wait for the update ---------------------------------------------------------
        if(heldList) {
            const unsigned int a = numDelays - 1u;
            deliver.addHeld(held, front);
            deliver.runs(heldList, a, heldCount, warp + warps, front);
            if(L.kind[a] == RESIDENT_LATE) deliver.spans(heldList, a, heldCount, 1u, front);
        }
        if constexpr(ONE) front.advance();
        else {
            #pragma unroll
            for(unsigned int c = 0; c < RESIDENT_CLASSES; c++) {
                if(c < L.num_depths) front.f[c] = (front.f[c] + 1u == L.depth[c]) ? 0u : front.f[c] + 1u;
            }
        }
        buf = (buf + 1u == L.buffers) ? 0u : buf + 1u;
        histAt = (histAt + 1u == L.history) ? 0u : histAt + 1u;
        if(++recAt == (unsigned int)L.neuron.num_recording_timesteps) recAt = 0u;
        // (a lane adds far less than 2^31 events in a step: that many synapses of one CTA do not fit the device)
        if(L.count_events && (deliver.events >> 24)) {
            atomicAdd(&state->synaptic_events, (unsigned long long)deliver.events);
            deliver.events = 0u;
        }
        if(step + 1u == sh.steps) break;
    }

ended: __attribute__((unused));
    // ---------------- what the launch leaves in memory ----------------------------------------------------
    // every CTA is through its last step: nobody reads the spike lists any more
    const unsigned int step = sh.steps;
    const unsigned long long doneNow = sh.done + step;
    const unsigned int k = (sh.phase + step) % sh.period, period = sh.period;
    __syncthreads();
    // (A launch of one step fills one list, which the step before it has emptied: only the counters wait for the other CTAs.  The
    // hand-shake took 1 us of such a launch.)
    const bool single = step == 1u;
    if(asked < G && (!single || me == 0)) awaitCell(buf == 0u ? L.buffers - 1u : buf - 1u, no0 + step, &sh.stop[turn]);
    __syncthreads();
    if(sh.stop[turn] & 1u) return;
    // lists of the last steps: emptied by the first CTA (and the one the next step writes), filled by all
    const unsigned int lists = min(L.history, step);
    if(me == 0) {
        for(unsigned int i = threadIdx.x; i < numGroups * (single ? 1u : lists + 1u); i += blockDim.x) {
            const b200_neuron_group &g = groups[i % numGroups];
            const unsigned int t = i / numGroups;      // 0: the next step, t: t - 1 steps ago
            if(t < g.num_delay_slots) g.spk_cnt[ringSlot(k + 1u + g.num_delay_slots - t, g.num_delay_slots)] = 0u;
        }
        __threadfence();
        __syncthreads();
        if(threadIdx.x == 0) storeRelaxedGpu(L.leave, L.launch);
    }
    else if(!single) {
        if(threadIdx.x == 0) {
            unsigned int polls = 0;
            while(loadRelaxedGpu(L.leave) != L.launch && !gaveUp(polls, &sh.stop[turn])) {}
            __threadfence();
        }
        __syncthreads();
    }
    if(mine) {
        const b200_neuron_group &g = groups[group];
        for(unsigned int t = 0; t < lists && t + 1u < g.num_delay_slots; t++) {
            const unsigned int b = residentTable<const unsigned int>(L.at.history)[((histAt + 2u * L.history - 1u - t) % L.history) * RESIDENT_UNITS + warp];
            if(!b) continue;
            const unsigned int slot = ringSlot(k + period - t, g.num_delay_slots);
            unsigned int at = 0;
            if(lane == 0) at = atomicAdd(&g.spk_cnt[slot], __popc(b));
            at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(b & ((1u << lane) - 1u));
            if((b >> lane) & 1u) {
                if(at < g.num_neurons) g.spk[(size_t)slot * g.num_neurons + at] = local;
                else atomicOr(&state->error, ERR_SPIKE_OVERFLOW);
            }
        }
    }
    if(mine && active) {
        const b200_neuron_group &g = groups[group];
        storeNeuron(g, local, regs, false);
        #pragma unroll
        for(unsigned int p = 0; p < NPSM; p++) {
            if(p < g.num_psm && g.psm[p].max_den_delay) {
                const unsigned int c = myCol[p] >> 24, n = sh.columns[c];
                const float *cell = acc + (myCol[p] & 0xFFFFFFu);
                float *ring = g.psm[p].den_delay + local;
                #pragma unroll 8
                for(unsigned int d = 0; d < sh.depth[c]; d++) ring[(size_t)d * g.num_neurons] = cell[d * n];
            }
        }
    }
    if(L.count_events) {
        // (halves, so that the sum over a warp does not pass 32 bits)
        const unsigned long long e = __reduce_add_sync(0xFFFFFFFFu, deliver.events & 0xFFFFu) +
                                     ((unsigned long long)__reduce_add_sync(0xFFFFFFFFu, deliver.events >> 16) << 16);
        if(lane == 0 && e) atomicAdd(&state->synaptic_events, e);
        if(spikes) atomicAdd(&state->spikes, (unsigned long long)spikes);
    }
    // (every CTA has sent the message of the last step, so every CTA has read the counters)
    if(me == 0 && threadIdx.x == 0) {
        state->timestep = t0 + step;
        state->steps_done = doneNow;
        state->phase = k;
        const unsigned int quiet = (step > sh.accounted) ? min(step - sh.accounted, 1u << 14) : 0u;
        residentSettle(L, *state, max(sh.debt - (int)(quiet * (L.spare / 2u)), 0), step, doneNow);
    }
}

// Kernel instances of one compilation unit.
template<bool ONE, unsigned int BLOCK>
inline const void *residentInstance(int npsm, int ncs)
{
#define B200_RESIDENT(P, C) if(npsm == P && ncs == C) return (const void*)residentStepKernel<P, C, ONE, BLOCK>
    B200_RESIDENT(1, 0); B200_RESIDENT(1, 1); B200_RESIDENT(1, B200_MAX_CS);
    B200_RESIDENT(2, 0); B200_RESIDENT(2, 1); B200_RESIDENT(2, B200_MAX_CS);
    B200_RESIDENT(B200_MAX_PSM, 0); B200_RESIDENT(B200_MAX_PSM, 1); B200_RESIDENT(B200_MAX_PSM, B200_MAX_CS);
#undef B200_RESIDENT
    return nullptr;
}
}   // namespace b200
