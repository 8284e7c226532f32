// Neuron update kernel: postsynaptic models, current sources, neuron dynamics,
// threshold, reset, spike emission and recording for every merged neuron group
// in one launch.  Replaces the reference's neuronSpikeQueueUpdateKernel +
// updateNeuronsKernel pair (backendSIMT.cc:373-662) and the per-group code of
// NeuronUpdateGroupMerged::generateNeuronUpdate
// (neuronUpdateGroupMerged.cc:552-773).
//
// Layout: one thread per neuron, groups padded to whole blocks, grid.y = batch.
// All state is SoA fp32 so every load/store is a coalesced 128-byte line per
// warp.  Spikes are compacted with a warp ballot and ONE atomicAdd per warp
// that spiked (the reference stages ids in shared memory and issues one atomic
// per block per step whether or not anything spiked).  The same ballot word is
// the 32-neuron spike-recording word, written with a plain store.  The last
// block to finish (ticket) clears the spike counts of the slot the next step
// will write and advances the step counters, which is what the reference's
// separate one-thread-per-group queue-update kernel does.
//
// Arithmetic uses single IEEE operations without fused contraction in the
// order of the reference's model strings (neuronModels.h:168-241,
// postsynapticModels.h:98-148, currentSourceModels.h:111-122) so results are
// bit-identical to the CPU backend for identical inputs.
#pragma once

#include "common.cuh"

namespace b200
{
constexpr int NEURON_BLOCK = 128;
constexpr unsigned int NEURON_BLOCKS_PER_SM = 16;
constexpr unsigned int NEURON_STAGED = 8;           // most groups whose tables a block takes into shared memory
constexpr unsigned int NEURON_STAGED_ANY = 4;       // as many however large the launch and whatever kernel runs before it
// Warps of an SM before a warp takes four words of neurons.  us a step of a network of 80 000 / 150 000 / 200 000 / 300 000 / 1 200 000
// neurons with one word a warp 4.4 / 4.7 / 6.7 / 7.4 / 15.1, with four 5.3 / 5.6 / 5.5 / 5.5 / 11.9; with a Poisson source each 5.3 / 5.6 /
// 8.0 / 9.0 / 21.7 and 7.2 / 8.1 / 8.2 / 7.9 / 21.8: the line, 152 000 neurons, is where the second wave of blocks begins.
constexpr unsigned int NEURON_WARPS_WANTED = 8;

// Peers of a sharded model as the neuron update sees them: every spike id is also
// stored into each peer's exchange arena, at the offset it has in this process's.
struct ExchangeCtx
{
    unsigned int world;
    unsigned int rank;
    unsigned char *arena;
    unsigned char *const *peers;        // [B200_MAX_RANKS], shared or global memory
    unsigned long long tag;             // step number the words of this step carry in their high half
};

struct NeuronLaunch
{
    const b200_neuron_group *groups;
    const unsigned int *block_start;
    unsigned int num_groups;
    unsigned int batch;
    float dt;
    unsigned long long seed;
    unsigned long long num_recording_timesteps;
    StepState *state;
    unsigned int count_events;
    unsigned int ahead;                 // steps of this block of steps that come before this one
    unsigned int advance;               // last kernel of a block of steps: how many it has, else 0
    unsigned long long peak_groups = ~0ull;     // which of the first 64 groups' spikes count for StepState::peak_spikes
};

// Loads of data other SMs write between grid barriers (postsynaptic input,
// spike times) must come from L2 when the kernel persists across time steps.
template<bool COHERENT, typename T>
__device__ __forceinline__ T loadShared(const T *p)
{
    return COHERENT ? __ldcg(p) : *p;
}

// Everything one neuron carries from step to step, as registers: the model's
// two state variables (bit patterns: SpikeSourceArray keeps integers), the
// running input of each fused postsynaptic model and each current source's
// variable.  Loading it as one batch of independent loads, before any store,
// keeps a single memory round trip on the critical path; the persistent kernel
// keeps it in registers across steps.
// NPSM / NCS bound the number of fused postsynaptic models and current sources
// of any group the kernel instance handles: the host picks the smallest
// instance that covers the model, so the unrolled loops below carry no dead
// iterations (a Potjans group has one of each).
template<int NPSM, int NCS>
struct NeuronRegs
{
    unsigned int v[2];
    float lin[NPSM];
    float cs[NCS > 0 ? NCS : 1];
};

__device__ __forceinline__ bool modelHasVar1(unsigned int model)
{
    return model != B200_NEURON_POISSON;
}

template<bool COHERENT, int NPSM, int NCS>
__device__ __forceinline__ void loadNeuron(const b200_neuron_group &g, unsigned long long bi, NeuronRegs<NPSM, NCS> &r)
{
    r.v[0] = static_cast<const unsigned int*>(g.vars[0])[bi];
    r.v[1] = modelHasVar1(g.model) ? static_cast<const unsigned int*>(g.vars[1])[bi] : 0u;
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        r.lin[p] = (p < g.num_psm) ? loadShared<COHERENT>(&g.psm[p].out_post[bi]) : 0.0f;
    }
    #pragma unroll
    for(unsigned int c = 0; c < NCS; c++) {
        r.cs[c] = (c < g.num_cs && g.cs[c].var0) ? g.cs[c].var0[bi] : 0.0f;
    }
}

template<int NPSM, int NCS>
__device__ __forceinline__ void storeNeuron(const b200_neuron_group &g, unsigned long long bi,
                                            const NeuronRegs<NPSM, NCS> &r, bool onlyPrivate)
{
    static_cast<unsigned int*>(g.vars[0])[bi] = r.v[0];
    if(modelHasVar1(g.model) && g.model != B200_NEURON_SPIKE_SOURCE_ARRAY) static_cast<unsigned int*>(g.vars[1])[bi] = r.v[1];
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        // inputs without a dendritic-delay ring receive reductions directly and
        // are written back every step by the caller
        if(p < g.num_psm && (!onlyPrivate || g.psm[p].max_den_delay)) g.psm[p].out_post[bi] = r.lin[p];
    }
    #pragma unroll
    for(unsigned int c = 0; c < NCS; c++) {
        if(c < g.num_cs && g.cs[c].var0) g.cs[c].var0[bi] = r.cs[c];
    }
}

// Front slot of every dendritic-delay ring: read and cleared
// (neuronUpdateGroupMerged.cc:96-113).
template<bool COHERENT, int NPSM>
__device__ __forceinline__ void takeFronts(const b200_neuron_group &g, unsigned int b, unsigned int i,
                                           unsigned int k, float (&front)[NPSM])
{
    // every load before any store: the pointers are generic, so a store between
    // two loads would force the second load to wait for the first
    float *slot[NPSM];
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        front[p] = 0.0f;
        slot[p] = nullptr;
        if(p < g.num_psm) {
            const unsigned int D = g.psm[p].max_den_delay;
            if(D) {
                slot[p] = &g.psm[p].den_delay[((unsigned long long)b * D + ringSlot(k + 1, D)) * g.num_neurons + i];
                front[p] = loadShared<COHERENT>(slot[p]);
            }
        }
    }
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        if(slot[p]) *slot[p] = 0.0f;
    }
}

// One neuron, one time step, entirely in registers.  Returns whether it spiked.
// Random draws of the current sources for one neuron and step: the number of
// Poisson events of each PoissonExp source.  They depend on nothing the
// presynaptic phase produces, so the persistent kernel computes them while the
// barrier after that phase is in flight.
// The model draws its Poisson count by multiplying uniforms until the product
// falls below exp(-lambda) (currentSourceModels.h:111-118); here the same count
// comes from inverting the Poisson CDF with one uniform, a quarter of a Philox
// block per step instead of one or two whole blocks.
template<int NCS>
__device__ __forceinline__ void drawCurrentSources(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b,
                                                   unsigned int i, unsigned long long timestep,
                                                   unsigned int (&count)[NCS > 0 ? NCS : 1])
{
    #pragma unroll
    for(unsigned int c = 0; c < NCS; c++) {
        count[c] = 0;
        if(c < g.num_cs && g.cs[c].model == B200_CS_POISSON_EXP) {
            const b200_current_source &cs = g.cs[c];
            const b200_philox_out blk = b200_rng_step_block(L.seed, cs.rng_stream, b * g.num_neurons + i, timestep);
            const float u = b200_u32_to_uniform(b200_rng_step_word(&blk, timestep));
            count[c] = b200_poisson_inverse(u, cs.params[2], cs.params[3]);
        }
    }
}

// Time to the next spike of a Poisson neuron that has none left (neuronModels.h:318-325): depends on nothing a step
// delivers, so the target-resident kernel draws it while it waits for the step's spikes.
__device__ __forceinline__ float drawPoissonInterval(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b, unsigned int i,
                                                     unsigned long long timestep, float tts)
{
    b200_rng rng = b200_rng_sim(L.seed, g.rng_stream, b * g.num_neurons + i, timestep);
    return B200_FADD(tts, B200_FMUL(g.params[0], -b200_logf(b200_rng_uniform(&rng))));
}

// WORDS neurons of a thread, 32 apart: what they share (the group's parameters, every branch) is done once for all, and their
// arithmetic chains run side by side.  Neurons that are not `active` are computed on whatever they hold and never spike.
template<int NPSM, int NCS, int WORDS>
__device__ __forceinline__ void neuronComputeWords(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b,
                                                   const unsigned int (&i)[WORDS], const bool (&active)[WORDS],
                                                   unsigned long long timestep, float t,
                                                   NeuronRegs<NPSM, NCS> (&r)[WORDS], const float (&front)[WORDS][NPSM],
                                                   const unsigned int (&csCount)[WORDS][NCS > 0 ? NCS : 1], bool (&spiked)[WORDS],
                                                   bool intervalDrawn = false)
{
    const unsigned int model = g.model;
    float Isyn[WORDS], V[WORDS];
    #pragma unroll
    for(int w = 0; w < WORDS; w++) {
        Isyn[w] = 0.0f;
        V[w] = __uint_as_float(r[w].v[0]);
        spiked[w] = false;
    }

    // incoming fused postsynaptic models
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        if(p < g.num_psm) {
            const b200_psm &psm = g.psm[p];
            float linSyn[WORDS];
            #pragma unroll
            for(int w = 0; w < WORDS; w++) linSyn[w] = psm.max_den_delay ? B200_FADD(r[w].lin[p], front[w][p]) : r[w].lin[p];
            if(psm.model == B200_PSM_EXP_CURR) {
                const float init = psm.params[0], decay = psm.params[1];
                #pragma unroll
                for(int w = 0; w < WORDS; w++) {
                    Isyn[w] = B200_FADD(Isyn[w], B200_FMUL(init, linSyn[w]));
                    r[w].lin[p] = B200_FMUL(linSyn[w], decay);
                }
            }
            else if(psm.model == B200_PSM_EXP_COND) {
                const float decay = psm.params[0], E = psm.params[1];
                #pragma unroll
                for(int w = 0; w < WORDS; w++) {
                    Isyn[w] = B200_FADD(Isyn[w], B200_FMUL(linSyn[w], B200_FSUB(E, V[w])));
                    r[w].lin[p] = B200_FMUL(linSyn[w], decay);
                }
            }
            else {
                #pragma unroll
                for(int w = 0; w < WORDS; w++) {
                    Isyn[w] = B200_FADD(Isyn[w], linSyn[w]);
                    r[w].lin[p] = 0.0f;
                }
            }
        }
    }

    // current sources
    #pragma unroll
    for(unsigned int c = 0; c < NCS; c++) {
        if(c < g.num_cs) {
            const b200_current_source &cs = g.cs[c];
            const float scale = cs.params[0], decay = cs.params[1];
            if(cs.model == B200_CS_DC) {
                #pragma unroll
                for(int w = 0; w < WORDS; w++) Isyn[w] = B200_FADD(Isyn[w], scale);
            }
            else {
                #pragma unroll
                for(int w = 0; w < WORDS; w++) {
                    const float current = B200_FADD(r[w].cs[c], B200_FMUL(scale, (float)csCount[w][c]));
                    Isyn[w] = B200_FADD(Isyn[w], current);
                    r[w].cs[c] = B200_FMUL(current, decay);
                }
            }
        }
    }

    if(model == B200_NEURON_LIF) {
        const float threshold = g.params[0], reset = g.params[1], rest = g.params[2], offset = g.params[3], rm = g.params[4],
                    decay = g.params[5], refractory = g.params[6];
        #pragma unroll
        for(int w = 0; w < WORDS; w++) {
            float R = __uint_as_float(r[w].v[1]);
            if(R <= 0.0f) {
                const float alpha = B200_FADD(B200_FMUL(B200_FADD(Isyn[w], offset), rm), rest);
                V[w] = B200_FSUB(alpha, B200_FMUL(decay, B200_FSUB(alpha, V[w])));
            }
            else {
                R = B200_FSUB(R, L.dt);
            }
            if(R <= 0.0f && V[w] >= threshold) {
                spiked[w] = active[w];
                V[w] = reset;
                R = refractory;
            }
            r[w].v[0] = __float_as_uint(V[w]);
            r[w].v[1] = __float_as_uint(R);
        }
    }
    else if(model == B200_NEURON_IZHIKEVICH) {
        const float a = g.params[0], bb = g.params[1], c = g.params[2], d = g.params[3];
        const float dt = L.dt;
        #pragma unroll
        for(int w = 0; w < WORDS; w++) {
            float U = __uint_as_float(r[w].v[1]), v = V[w];
            if(v >= 30.0f) {
                v = c;
                U = B200_FADD(U, d);
            }
            for(int half = 0; half < 2; half++) {
                // 0.04*V*V + 5*V + 140 - U + Isyn, left to right
                float x = B200_FMUL(B200_FMUL(0.04f, v), v);
                x = B200_FADD(x, B200_FMUL(5.0f, v));
                x = B200_FADD(x, 140.0f);
                x = B200_FSUB(x, U);
                x = B200_FADD(x, Isyn[w]);
                v = B200_FADD(v, B200_FMUL(B200_FMUL(0.5f, x), dt));
            }
            U = B200_FADD(U, B200_FMUL(B200_FMUL(a, B200_FSUB(B200_FMUL(bb, v), U)), dt));
            if(v > 30.0f) v = 30.0f;
            spiked[w] = active[w] && (v >= 29.99f);
            r[w].v[0] = __float_as_uint(v);
            r[w].v[1] = __float_as_uint(U);
        }
    }
    else if(model == B200_NEURON_SPIKE_SOURCE_ARRAY) {
        #pragma unroll
        for(int w = 0; w < WORDS; w++) {
            const unsigned int start = r[w].v[0], end = r[w].v[1];
            if(active[w] && start != end && t >= __ldg(&g.egp[start])) {
                spiked[w] = true;
                r[w].v[0] = start + 1;
            }
        }
    }
    else {
        #pragma unroll
        for(int w = 0; w < WORDS; w++) {
            float tts = V[w];
            if(active[w] && tts <= 0.0f && !intervalDrawn) tts = drawPoissonInterval(L, g, b, i[w], timestep, tts);
            tts = B200_FSUB(tts, 1.0f);
            spiked[w] = active[w] && (tts <= 0.0f);
            r[w].v[0] = __float_as_uint(tts);
        }
    }
}

template<int NPSM, int NCS>
__device__ __forceinline__ bool neuronCompute(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b,
                                              unsigned int i, unsigned long long timestep, float t,
                                              NeuronRegs<NPSM, NCS> &r, const float (&front)[NPSM],
                                              const unsigned int (&csCount)[NCS > 0 ? NCS : 1], bool intervalDrawn = false)
{
    const unsigned int one[1] = {i};
    const bool active[1] = {true};
    bool spiked[1];
    NeuronRegs<NPSM, NCS> regs[1] = {r};
    float fronts[1][NPSM];
    unsigned int counts[1][NCS > 0 ? NCS : 1];
    #pragma unroll
    for(int p = 0; p < NPSM; p++) fronts[0][p] = front[p];
    #pragma unroll
    for(int c = 0; c < (NCS > 0 ? NCS : 1); c++) counts[0][c] = csCount[c];
    neuronComputeWords<NPSM, NCS, 1>(L, g, b, one, active, timestep, t, regs, fronts, counts, spiked, intervalDrawn);
    r = regs[0];
    return spiked[0];
}

// Spike emission (ballot + one atomic per spiking warp), spike times and
// recording.  Called by whole warps.
template<bool COHERENT>
__device__ __forceinline__ void neuronEmit(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b,
                                           unsigned int local, bool spiked, unsigned int k,
                                           unsigned long long timestep, float t, const ExchangeCtx *x = nullptr)
{
    const unsigned int N = g.num_neurons;
    const unsigned int i = g.first_neuron + local;
    const bool active = local < g.num_update;
    const unsigned int slots = g.num_delay_slots;
    const unsigned int wslot = ringSlot(k + 1, slots);
    const unsigned int listStride = g.spk_slot_stride ? g.spk_slot_stride : N;
    const unsigned int ballot = __ballot_sync(0xFFFFFFFFu, spiked);
    const unsigned int lane = threadIdx.x & 31u;
    if(ballot) {
        unsigned int base = 0;
        if(lane == 0) {
            base = atomicAdd(&g.spk_cnt[b * slots + wslot], __popc(ballot));
        }
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if(L.count_events && lane == 0) atomicAdd(&L.state->spikes, (unsigned long long)__popc(ballot));
        if(spiked) {
            const unsigned int pos = base + __popc(ballot & ((1u << lane) - 1u));
            if(pos < listStride) {
                unsigned int *cell = &g.spk[((unsigned long long)b * slots + wslot) * listStride + pos];
                *cell = i;
                if(x) {
                    // the travelling copy: (step << 32 | id) into the same cell of every
                    // process's arena, this one included.  Each word validates itself,
                    // so the stores need no ordering and nothing waits for them.
                    unsigned long long *wire = reinterpret_cast<unsigned long long*>(g.spk_wire) +
                                               ((unsigned long long)b * slots + wslot) * listStride + pos;
                    const unsigned long long word = (x->tag << 32) | (unsigned long long)i;
                    for(unsigned int p = 0; p < x->world; p++) {
                        unsigned long long *dst = (p == x->rank) ? wire
                            : reinterpret_cast<unsigned long long*>(x->peers[p] + (reinterpret_cast<unsigned char*>(wire) - x->arena));
                        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" :: "l"(dst), "l"(word) : "memory");
                    }
                }
            }
            else {
                atomicOr(&L.state->error, ERR_SPIKE_OVERFLOW);
            }
        }
    }
    // spike times ride in the queue: carry the previous slot forward
    if(g.spike_times && active) {
        float *st = g.spike_times + ((unsigned long long)b * slots) * N;
        st[(unsigned long long)wslot * N + i] = spiked ? t : loadShared<COHERENT>(&st[(unsigned long long)ringSlot(k, slots) * N + i]);
    }
    // recording: the updated slice only, bit j%32 of word j/32 for its j-th neuron
    // (backendSIMT.cc:617-660 for a whole population)
    if(g.record_spk && L.num_recording_timesteps) {
        const unsigned int words = (g.num_update + 31u) / 32u;
        // a warp covers exactly one word; only the writing lane pays for the 64-bit modulo
        if(lane == 0 && (local / 32u) < words) {
            unsigned int *rec = g.record_spk + ((timestep % L.num_recording_timesteps) * L.batch + b) * words;
            rec[local / 32u] = ballot;
        }
    }
}

// One neuron, one time step with its state in global memory: called by whole
// warps (`local` may lie past the end of the group; such lanes only take part in
// the ballot).  `k` is the number of completed steps, `timestep` the model step.
template<bool COHERENT, int NPSM, int NCS>
__device__ __forceinline__ void neuronStep(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b,
                                           unsigned int local, unsigned int k, unsigned long long timestep,
                                           const ExchangeCtx *x = nullptr)
{
    const unsigned int i = g.first_neuron + local;
    const float t = B200_FMUL((float)timestep, L.dt);
    bool spiked = false;
    if(local < g.num_update) {
        const unsigned long long bi = (unsigned long long)b * g.num_neurons + i;
        NeuronRegs<NPSM, NCS> r;
        float front[NPSM];
        unsigned int csCount[NCS > 0 ? NCS : 1];
        loadNeuron<COHERENT>(g, bi, r);
        takeFronts<COHERENT, NPSM>(g, b, i, k, front);
        drawCurrentSources<NCS>(L, g, b, i, timestep, csCount);
        spiked = neuronCompute(L, g, b, i, timestep, t, r, front, csCount);
        storeNeuron(g, bi, r, false);
    }
    neuronEmit<COHERENT>(L, g, b, local, spiked, k, timestep, t, x);
}

// A warp's WORDS x 32 neurons of one group, one time step with their state in global memory: every load before any store
// (the pointers are generic: a store between two loads would make the second wait), one place in the spike list for all.
template<int NPSM, int NCS, int WORDS>
__device__ __forceinline__ void neuronWords(const NeuronLaunch &L, const b200_neuron_group &g, unsigned int b, unsigned int firstLocal,
                                            unsigned int k, unsigned long long timestep)
{
    const unsigned int lane = threadIdx.x & 31u, N = g.num_neurons, update = g.num_update, slots = g.num_delay_slots;
    const unsigned int wslot = ringSlot(k + 1, slots);
    const float t = B200_FMUL((float)timestep, L.dt);
    NeuronRegs<NPSM, NCS> r[WORDS];
    float front[WORDS][NPSM], was[WORDS];
    unsigned int csCount[WORDS][NCS > 0 ? NCS : 1], i[WORDS];
    bool active[WORDS], spiked[WORDS];
    float *const times = g.spike_times ? g.spike_times + (unsigned long long)b * slots * N : nullptr;
    const unsigned int rslot = times ? ringSlot(k, slots) : 0u;
    #pragma unroll
    for(int w = 0; w < WORDS; w++) {
        const unsigned int local = firstLocal + 32u * w + lane;
        active[w] = local < update;
        i[w] = g.first_neuron + local;
        if(active[w]) {
            loadNeuron<false>(g, (unsigned long long)b * N + i[w], r[w]);
            if(times) was[w] = times[(unsigned long long)rslot * N + i[w]];
        }
    }
    // front slots of the dendritic-delay rings: read and cleared (neuronUpdateGroupMerged.cc:96-113)
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) {
        const unsigned int D = p < g.num_psm ? g.psm[p].max_den_delay : 0u;
        float *const slot = D ? &g.psm[p].den_delay[((unsigned long long)b * D + ringSlot(k + 1, D)) * N] : nullptr;
        #pragma unroll
        for(int w = 0; w < WORDS; w++) front[w][p] = (slot && active[w]) ? slot[i[w]] : 0.0f;
        if(slot) {
            #pragma unroll
            for(int w = 0; w < WORDS; w++) if(active[w]) slot[i[w]] = 0.0f;
        }
    }
    #pragma unroll
    for(int w = 0; w < WORDS; w++) drawCurrentSources<NCS>(L, g, b, i[w], timestep, csCount[w]);
    neuronComputeWords<NPSM, NCS, WORDS>(L, g, b, i, active, timestep, t, r, front, csCount, spiked);
    unsigned int ballot[WORDS], total = 0;
    #pragma unroll
    for(int w = 0; w < WORDS; w++) {
        ballot[w] = __ballot_sync(0xFFFFFFFFu, spiked[w]);
        total += __popc(ballot[w]);
    }
    unsigned int base = 0;
    if(total && lane == 0) {
        base = atomicAdd(&g.spk_cnt[b * slots + wslot], total);
        if(L.count_events) atomicAdd(&L.state->spikes, (unsigned long long)total);
    }
    // (the state on its way while the place in the list is fetched)
    #pragma unroll
    for(int w = 0; w < WORDS; w++) {
        if(active[w]) {
            storeNeuron(g, (unsigned long long)b * N + i[w], r[w], false);
            // spike times ride in the queue: carry the previous slot forward
            if(times) times[(unsigned long long)wslot * N + i[w]] = spiked[w] ? t : was[w];
        }
    }
    // recording: bit j%32 of word j/32 for the group's j-th neuron (backendSIMT.cc:617-660 for a whole population)
    if(g.record_spk && L.num_recording_timesteps) {
        const unsigned int words = (update + 31u) / 32u;
        unsigned int *const rec = g.record_spk + ((timestep % L.num_recording_timesteps) * L.batch + b) * words + firstLocal / 32u;
        #pragma unroll
        for(int w = 0; w < WORDS; w++) if(lane == 0 && firstLocal / 32u + w < words) rec[w] = ballot[w];
    }
    if(total) {
        const unsigned int listStride = g.spk_slot_stride ? g.spk_slot_stride : N;
        unsigned int *const list = g.spk + ((unsigned long long)b * slots + wslot) * listStride;
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        #pragma unroll
        for(int w = 0; w < WORDS; w++) {
            if(spiked[w]) {
                const unsigned int pos = base + __popc(ballot[w] & ((1u << lane) - 1u));
                if(pos < listStride) list[pos] = i[w];
                else atomicOr(&L.state->error, ERR_SPIKE_OVERFLOW);
            }
            base += __popc(ballot[w]);
        }
    }
}

// WORDS = 4: a warp takes the 128 neurons of a padded block, a quarter of the instructions for each, as long as that leaves
// every SM its warps; WORDS = 1: a warp takes 32, for small networks, where the chain of one neuron is all there is.
// Whether the blocks of a launch take the tables of their groups (0.6 KB each) into shared memory ahead of chainWait().  The kernels before
// and behind use next to none of it, and where they and this one split an SM's memory differently, blocks of one are not placed beside
// those of the other: with room for eight groups in every block (5 KB) a step of two populations of 400 and 500 neurons with 32 copies took
// 7.6 us (DENSE) and 11.1 (STDP), without 7.2 and 10.7, with room for its own two 6.3 and 10.2.  us a step without / with, by groups and
// blocks: 2 to 4 groups, 10 to 2048 blocks: 6.1 / 5.2 to 11.1 / 10.3, at worst 11.3 / 11.4.  5 to 8 groups, DENSE: 25 blocks 6.5 / 5.5,
// 120 6.6 / 5.7, 200 7.0 / 7.0, 512 7.7 / 8.0, 728 7.8 / 8.4, 896 8.6 / 8.3, 1248 9.4 / 8.4, 4608 19.1 / 17.5; SPARSE: 25 blocks 6.7 / 5.6,
// 400 8.8 / 8.1, 512 6.8 / 7.1, 728 7.1 / 6.8, 1248 9.1 / 8.3; STDP 10.7 / 10.1, 12.0 / 11.7, 10.9 / 10.7, 11.1 / 11.0, 12.5 / 12.0.
// `blocks`: of 128 neurons, of all copies.  `dense`: the kernel before is one of a DENSE or BITMASK group.
inline bool neuronStaged(unsigned int groups, unsigned long long blocks, unsigned int sms, bool dense)
{
    if(groups <= NEURON_STAGED_ANY) return true;
    return groups <= NEURON_STAGED && (!dense || blocks <= sms || blocks >= 7u * sms);
}

inline size_t neuronTableBytes(unsigned int groups) { return sizeof(b200_neuron_group) * groups + sizeof(unsigned int) * (groups + 1u); }

template<int NPSM, int NCS, int WORDS, bool STAGED>
__global__ void __launch_bounds__(NEURON_BLOCK)
neuronUpdateKernel(const NeuronLaunch L)
{
    constexpr unsigned int PARTS = NEURON_BLOCK / (32 * WORDS);         // warps of a padded block
    const b200_neuron_group *groups = L.groups;
    const unsigned int *blockStart = L.block_start;
    if constexpr(STAGED) {
        // (common.cuh: stageGroup)
        extern __shared__ __align__(16) unsigned char neuronTables[];
        b200_neuron_group *const table = reinterpret_cast<b200_neuron_group*>(neuronTables);
        unsigned int *const starts = reinterpret_cast<unsigned int*>(table + L.num_groups);
        // (small launches wait for the tables: one round trip.  Large ones, a pass of 20 steps and its fetches with loads / asynchronous
        // copies: batched SPARSE 20 000 + 20 000 with 8 copies 783 / 795 us, DENSE 6556 x 5007 with 16 765 / 775, 8192 x 8192 with 32 796 / 778)
        if constexpr(WORDS == 1) {
            stageWordsAsync(table, L.groups, sizeof(b200_neuron_group) * L.num_groups);
            stageWordsAsync(starts, L.block_start, sizeof(unsigned int) * (L.num_groups + 1u));
            stagedWords();
        }
        else {
            stageWords(table, L.groups, sizeof(b200_neuron_group) * L.num_groups);
            stageWords(starts, L.block_start, sizeof(unsigned int) * (L.num_groups + 1u));
        }
        __syncthreads();
        groups = table;
        blockStart = starts;
    }
    const unsigned int blocks = blockStart[L.num_groups], launched = gridDim.x * gridDim.y;
    const unsigned int rank = blockIdx.y * gridDim.x + blockIdx.x;
    chainWait();
    const unsigned int k = chainPhase(L.state, L.ahead);
    const unsigned long long timestep = L.state->timestep + L.ahead;
    for(unsigned int unit = rank * (NEURON_BLOCK / 32) + (threadIdx.x >> 5); unit < blocks * L.batch * PARTS; unit += launched * (NEURON_BLOCK / 32)) {
        const unsigned int item = unit / PARTS, b = item / blocks, block = item - b * blocks;
        const unsigned int gi = findGroup(blockStart, L.num_groups, block);
        neuronWords<NPSM, NCS, WORDS>(L, groups[gi], b, (block - blockStart[gi]) * NEURON_BLOCK + (unit % PARTS) * 32u * WORDS, k, timestep);
    }

    // ---- queue update for the next step: its slot was last read three steps ago at the latest -------
    if(rank == launched - 1u) {
        __shared__ unsigned int stepSpikes;
        if(threadIdx.x == 0) stepSpikes = 0u;
        __syncthreads();
        for(unsigned int q = threadIdx.x; q < L.num_groups * L.batch; q += blockDim.x) {
            const b200_neuron_group &o = groups[q / L.batch];
            const unsigned int ob = q % L.batch;
            // (the spikes of the step before: this one's are not all there yet)
            if(q / L.batch >= 64u || ((L.peak_groups >> (q / L.batch)) & 1ull)) {
                atomicAdd(&stepSpikes, o.spk_cnt[ob * o.num_delay_slots + ringSlot(k, o.num_delay_slots)]);
            }
            o.spk_cnt[ob * o.num_delay_slots + ringSlot(k + 2, o.num_delay_slots)] = 0;
        }
        __syncthreads();
        if(threadIdx.x == 0 && stepSpikes) atomicMax(&L.state->peak_spikes, stepSpikes);
    }
    // ---- behind a block of steps: the counters, once every block has read them ------------------------
    if(L.advance) {
        __syncthreads();
        if(threadIdx.x == 0 && atomicAdd(&L.state->ticket, 1u) == launched - 1u) {
            L.state->ticket = 0;
            L.state->timestep = timestep + 1;
            L.state->steps_done = L.state->steps_done + L.advance;
            L.state->phase = (k + 1 == L.state->ring_period) ? 0u : k + 1;
        }
    }
}
}   // namespace b200
