// Time steps of the target-resident path in windows.
//
// Where no spike of a window of steps reaches any neuron within that window, the chain neuron update -> spikes -> synapses ->
// neuron update (resident.h) does not go through another SM in every step, only in every window:
//
//   LATE  one axonal delay of a steps for all groups, no ring: windows of a + 1 steps, or of a whole part of that;
//   FEED  all spikes come from populations without inputs (Poisson neurons, spike source arrays).  Those are updated a window
//         ahead of the others, so that their spikes are there when they are wanted.
//
// Units of 32 neurons, the private copy of the synapses and the tables are those of residentStepKernel, and memory is left as that
// leaves it.  A window: the CTAs' messages (a head with a tag and a count, 16-bit entries: step, unit, neuron) become a list of
// spikes for every step; all of them are added to input buffers in shared memory, one for each step of the window; then each warp
// takes its 32 neurons through all steps on its own.  Two or three barriers of a CTA a window instead of a step, loads of a
// window's runs side by side instead of a step's, and the wait for the messages once (FEED: hidden behind a window).
//
// us a step of calls of 2000, step by step / in windows: 1000 sources -> 10 000 neurons, p = 0.1, 2 spikes a step 2.19 / 0.26; BITMASK
// 2003 -> 5009, 80 spikes 3.75 / 0.49; DENSE 4096 x 4096, 100 spikes 3.88 / 0.85; 100 000 neurons with conductances, delay 10 2.67 / 1.32.
// Cycles of a window of the last two: deliveries 7400 and 3500, updates 1000 and 5000, messages 4800 - 8500 and 9800.
#pragma once

#include "resident_step.cuh"

namespace b200
{
struct WindowShared
{
    unsigned int count[2][32];          // spikes of each step of the window (counts on beyond the list's end): of even and odd windows
    unsigned int sent[2];               // entries of the message that is being made, of even and odd ones
    unsigned short first[2][4];         // and the first of them
    unsigned int stop;                  // 1: a wait ran out, 4: more spikes than the list holds
    unsigned int steps;                 // of this launch
    int debt;
    unsigned int phase, period, limit;
    unsigned long long done;
    unsigned int firstWarp[RESIDENT_MAX_GROUPS + 1];
    __align__(16) ResidentLif lif[RESIDENT_MAX_GROUPS];
};

__device__ __forceinline__ void fenceGpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Spikes [from, to) of a step's list through a DENSE or BITMASK group onto 32 targets: a lane's sum.  (The whole warp calls; `from`
// and the list are multiples of four entries.)  `mixed`: the list has spikes of other populations too.  A row's part is 128 bytes out
// of L2 and an addition, so instructions count: with every choice made for every spike there were 49 for one, and a step of DENSE
// 4096 x 4096 with 100 spikes took 0.27 us longer.
__device__ __forceinline__ float windowSpan(const ResidentSpan &S, const unsigned int *list, unsigned int from, unsigned int to, unsigned int unit, bool mixed, unsigned int &events)
{
    const unsigned int lane = threadIdx.x & 31u, post = unit * 32u + lane, src = S.src_group, numTrg = S.num_trg;
    const float weight = S.weight;
    const bool valid = post < numTrg;
    float sum = 0.0f;
    unsigned int n = 0;
    if(const unsigned int *const gp = S.gp) {
        constexpr unsigned int SIDE = 4;            // words of a lane in flight
        const unsigned int rowWords = S.row_stride / 32u;
        for(; from < to; from += 32u * SIDE) {
            unsigned int word[SIDE];
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) {
                const unsigned int at = from + u * 32u + lane, spike = (at < to) ? list[at] : 0xFFFFFFFFu;
                word[u] = 0u;
                if((spike >> 24) == src) word[u] = __ldg(gp + (unsigned long long)(spike & 0xFFFFFFu) * rowWords + unit);
            }
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) {
                if(from + u * 32u >= to) break;
                // 32 x 32 bits across the warp, rows and columns exchanged (halves, quarters, ...): bit i of lane b is then bit
                // 31 - b of lane i's word
                unsigned int c = __brev(word[u]), low = 0x0000FFFFu;
                #pragma unroll
                for(unsigned int o = 16; o; o >>= 1, low ^= low << o) {
                    const unsigned int v = __shfl_xor_sync(0xFFFFFFFFu, c, o);
                    c = (lane & o) ? ((c & ~low) | ((v >> o) & low)) : ((c & low) | ((v << o) & ~low));
                }
                n += __popc(c);
            }
        }
        if(valid) {
            events += n;
            sum = (float)n * weight;
        }
        return sum;
    }
    const float *const g = S.g;
    if(g && !mixed) {
        // (lanes beyond the targets read the last one's weights)
        constexpr unsigned int LOADS = 16;
        const char *const base = reinterpret_cast<const char*>(g + min(post, numTrg - 1u));
        const unsigned int rowBytes = numTrg * (unsigned int)sizeof(float);
        n = to - from;
        for(; from + LOADS <= to; from += LOADS) {
            float w[LOADS];
            #pragma unroll
            for(unsigned int u = 0; u < LOADS; u += 4u) {
                const uint4 s4 = *reinterpret_cast<const uint4*>(list + from + u);
                w[u] = __ldg(reinterpret_cast<const float*>(base + (unsigned long long)(s4.x & 0xFFFFFFu) * rowBytes));
                w[u + 1u] = __ldg(reinterpret_cast<const float*>(base + (unsigned long long)(s4.y & 0xFFFFFFu) * rowBytes));
                w[u + 2u] = __ldg(reinterpret_cast<const float*>(base + (unsigned long long)(s4.z & 0xFFFFFFu) * rowBytes));
                w[u + 3u] = __ldg(reinterpret_cast<const float*>(base + (unsigned long long)(s4.w & 0xFFFFFFu) * rowBytes));
            }
            #pragma unroll
            for(unsigned int u = 0; u < LOADS; u++) sum += w[u];
        }
        for(; from < to; from += 4u) {
            float w[4];
            #pragma unroll
            for(unsigned int u = 0; u < 4u; u++) {
                w[u] = 0.0f;
                if(from + u < to) w[u] = __ldg(reinterpret_cast<const float*>(base + (unsigned long long)(list[from + u] & 0xFFFFFFu) * rowBytes));
            }
            sum += (w[0] + w[1]) + (w[2] + w[3]);
        }
    }
    else {
        constexpr unsigned int LOADS = RESIDENT_DENSE_SPIKES;
        for(; from < to; from += LOADS) {
            float w[LOADS];
            #pragma unroll
            for(unsigned int u = 0; u < LOADS; u++) {
                const unsigned int spike = (from + u < to) ? list[from + u] : 0xFFFFFFFFu;
                const bool take = (spike >> 24) == src && valid;
                w[u] = (take && !g) ? weight : 0.0f;
                if(take && g) w[u] = __ldg(&g[(unsigned long long)(spike & 0xFFFFFFu) * numTrg + post]);
                n += take ? 1u : 0u;
            }
            #pragma unroll
            for(unsigned int u = 0; u < LOADS; u++) sum += w[u];
        }
    }
    if(!valid) return 0.0f;
    events += n;
    return sum;
}

template<int NPSM, int NCS>
__global__ void __launch_bounds__(RESIDENT_BLOCK, 1)
residentWindowKernel(const __grid_constant__ ResidentWindowLaunch A)
{
    __shared__ WindowShared sh;
    const ResidentLaunch &L = A.L;
    const ResidentWindow &W = A.W;
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const unsigned int numGroups = L.neuron.num_groups, G = gridDim.x, me = blockIdx.x;
    const b200_neuron_group *const groups = residentTable<const b200_neuron_group>(L.at.groups);
    const unsigned int *const unitFirst = residentTable<const unsigned int>(L.at.unit_first);
    const ResidentRun *const runTable = residentTable<const ResidentRun>(L.at.runs);
    unsigned int *const list = residentTable<unsigned int>(W.list_at);
    unsigned int *const words = residentTable<unsigned int>(W.words_at);
    float *const acc = residentTable<float>(W.acc_at);
    stageWordsAsync(residentSmem + L.at.groups, L.neuron.groups, sizeof(b200_neuron_group) * numGroups);
    stageWordsAsync(residentSmem + L.at.unit_start, L.unit_start, sizeof(unsigned int) * (numGroups + 1));
    stageWordsAsync(residentSmem + L.at.unit_first, L.unit_first, sizeof(unsigned int) * L.num_units);
    stageWordsAsync(residentSmem + L.at.columns, L.columns + (size_t)me * RESIDENT_UNITS * B200_MAX_PSM, sizeof(unsigned int) * RESIDENT_UNITS * B200_MAX_PSM);
    stageWordsAsync(residentSmem + L.at.runs, L.runs + (size_t)me * numGroups, sizeof(ResidentRun) * numGroups);
    stageWordsAsync(residentSmem + L.at.rows, L.rows, sizeof(unsigned long long) * numGroups);
    stageWordsAsync(residentSmem + L.at.spans, L.spans, sizeof(ResidentSpan) * L.num_spans);
    StepState *const state = L.neuron.state;
    const unsigned long long t0 = state->timestep;
    if(L.may_leave) {
        if(me == 0 && threadIdx.x == 0) *L.barrier = 0ull;
        if(state->steps_done < state->resident_hold) {              // (the same for every CTA: both change at the end of a launch)
            stagedWords();
            return;
        }
    }
    const unsigned int K = W.steps, delay = L.delay[0], columns = L.cta_columns[me * RESIDENT_CLASSES];
    if(threadIdx.x == 0) {
        sh.debt = (int)state->resident_debt;
        sh.sent[0] = sh.sent[1] = 0u;
        for(int i = 0; i < 8; i++) sh.first[i / 4][i % 4] = 0u;
        sh.stop = 0u;
        sh.steps = L.num_steps;
        sh.done = state->steps_done;
        sh.phase = state->phase;
        sh.period = state->ring_period;
        sh.limit = (unsigned int)min(state->barrier_spin_limit, 0xFFFFFFFFull);
    }
    if(threadIdx.x < 32u) sh.count[0][threadIdx.x] = sh.count[1][threadIdx.x] = 0u;
    for(unsigned int i = threadIdx.x; i < K * columns; i += blockDim.x) acc[i] = 0.0f;
    for(unsigned int i = threadIdx.x; i < numGroups; i += blockDim.x) residentLifTable(sh.lif[i], L.neuron.groups[i]);
    stagedWords();
    __syncthreads();
    // (up to 65 entries; the option "resident_warps" allows blocks of 32 threads)
    for(unsigned int i = threadIdx.x; i <= numGroups; i += blockDim.x) {
        // first warp whose unit (warp * G + me) is not before the group
        const unsigned int u = residentTable<const unsigned int>(L.at.unit_start)[i];
        sh.firstWarp[i] = (u <= me) ? 0u : (u - me + G - 1u) / G;
    }

    // this thread's neuron
    const bool mine = warp < RESIDENT_UNITS && warp * G + me < L.num_units;
    unsigned int group = 0, local = 0, what = 0;
    bool active = false, ahead = false;     // ahead: of a population that is updated a window early
    float nextTime = 0.0f;
    NeuronRegs<NPSM, NCS> regs;
    unsigned int myCol[NPSM];
    #pragma unroll
    for(unsigned int p = 0; p < NPSM; p++) myCol[p] = 0u;
    if(mine) {
        group = unitFirst[warp * G + me] >> 24;
        local = (unitFirst[warp * G + me] & 0xFFFFFFu) + lane;
        const b200_neuron_group &g = groups[group];
        active = local < g.num_update;
        ahead = W.feed && ((W.free_groups >> group) & 1ull);
        what = residentWhat<NCS>(g, (L.source_groups >> group) & 1ull, false);
        #pragma unroll
        for(unsigned int p = 0; p < NPSM; p++) myCol[p] = (residentTable<const unsigned int>(L.at.columns)[warp * B200_MAX_PSM + p] & 0xFFFFu) + lane;
        if(active) {
            loadNeuron<true>(g, local, regs);
            if((what & RESIDENT_IS_ARRAY) && regs.v[0] != regs.v[1]) nextTime = __ldg(&g.egp[regs.v[0]]);
        }
    }
    // FEED: the warps without neurons read the messages, while the others update theirs.  LATE: as few as it takes, for nobody has
    // anything else to do, and the more ask for the heads, the longer each waits (100 000 neurons on 148 CTAs, five warps instead of
    // 24: 1.44 -> 1.38 us a step)
    const unsigned int neuronWarps = (L.num_units + G - 1u) / G;
    const unsigned int firstReader = !W.feed ? warps - (G + 31u) / 32u : (2u * neuronWarps <= warps && (warps - neuronWarps) * 32u >= G) ? neuronWarps : 0u;
    const unsigned int readers = warps - firstReader, perReader = (G + readers - 1u) / readers;
    const unsigned int recAt = L.neuron.num_recording_timesteps ? (unsigned int)(t0 % L.neuron.num_recording_timesteps) : 0u;
    unsigned int spikes = 0, events = 0;
    auto gaveUp = [&](unsigned int &polls) -> bool {
        if(++polls <= sh.limit) return false;
        atomicOr(&state->error, ERR_BARRIER_TIMEOUT);
        atomicOr(&sh.stop, 1u);
        return true;
    };
    auto tagOf = [&](unsigned int message) { return windowTag(W.epoch, message); };
    auto shortTagOf = [&](unsigned int message) { return windowShortTag(W.epoch, message); };

    // ---- the neurons of this warp through steps [first, first + n) of the launch; lane j gets the ballot of the j-th.
    // Populations without inputs: nothing to add up, and a Poisson neuron goes from spike to spike.
    auto freeSteps = [&](unsigned int first, unsigned int n) -> unsigned int {
        const b200_neuron_group &g = groups[group];
        unsigned int mask = 0, mineWord = 0;
        if(what & RESIDENT_IS_POISSON) {
            // The steps one by one take 1 off the time to the next spike, draw another when there is none left, and spike at 0 or
            // below.  Differences of a number of at least 1 and 1 are exact up to 2^24, so several steps are one.
            float left = __uint_as_float(regs.v[0]);
            for(unsigned int at = active ? 0u : n; at < n;) {
                if(left <= 0.0f) left = drawPoissonInterval(L.neuron, g, 0u, local, t0 + first + at, left);
                if(left > 0.0f && left < 16777216.0f) {
                    const unsigned int upTo = (unsigned int)ceilf(left);
                    if(upTo <= n - at) {
                        left = B200_FSUB(B200_FSUB(left, (float)(upTo - 1u)), 1.0f);
                        at += upTo;
                        mask |= 1u << (at - 1u);
                    }
                    else {
                        left = B200_FSUB(left, (float)(n - at));
                        at = n;
                    }
                }
                else {
                    left = B200_FSUB(left, 1.0f);
                    if(left <= 0.0f) mask |= 1u << at;
                    at++;
                }
            }
            __syncwarp();
            if(active) regs.v[0] = __float_as_uint(left);
        }
        else {
            for(unsigned int j = 0; j < n; j++) {
                if(active && regs.v[0] != regs.v[1] && B200_FMUL((float)(t0 + first + j), L.neuron.dt) >= nextTime) {
                    mask |= 1u << j;
                    if(++regs.v[0] != regs.v[1]) nextTime = __ldg(&g.egp[regs.v[0]]);
                }
            }
            __syncwarp();
        }
        for(unsigned int j = 0; j < n; j++) {
            const unsigned int word = __ballot_sync(0xFFFFFFFFu, (mask >> j) & 1u);
            if(lane == j) mineWord = word;
        }
        return mineWord;
    };
    auto fedSteps = [&](unsigned int first, unsigned int n) -> unsigned int {
        const b200_neuron_group &g = groups[group];
        unsigned int mineWord = 0;
        float *buffer = acc;
        if(what & RESIDENT_IS_LIF) {
            constexpr int INPUTS = NPSM < 2 ? NPSM : 2;
            constexpr unsigned int SIDE = 4;        // steps whose inputs are loaded together
            const ResidentLif q = sh.lif[group];    // (in registers: a store to shared memory would have it loaded again)
            for(unsigned int from = 0; from < n; from += SIDE) {
                float x[SIDE][NPSM];
                #pragma unroll
                for(unsigned int u = 0; u < SIDE; u++) {
                    #pragma unroll
                    for(int p = 0; p < NPSM; p++) {
                        x[u][p] = 0.0f;
                        if(p < INPUTS && (what & (p ? RESIDENT_HAS_TWO : RESIDENT_HAS_INPUT)) && from + u < n) x[u][p] = buffer[u * columns + myCol[p]];
                    }
                }
                #pragma unroll
                for(unsigned int u = 0; u < SIDE; u++) {
                    #pragma unroll
                    for(int p = 0; p < INPUTS; p++) {
                        if((what & (p ? RESIDENT_HAS_TWO : RESIDENT_HAS_INPUT)) && from + u < n) buffer[u * columns + myCol[p]] = 0.0f;
                    }
                }
                #pragma unroll
                for(unsigned int u = 0; u < SIDE; u++) {
                    if(from + u < n) {
                        const bool spiked = residentLif(q, L.neuron.dt, regs, x[u], what, 0u) && active;
                        const unsigned int word = __ballot_sync(0xFFFFFFFFu, spiked);
                        if(lane == from + u) mineWord = word;
                    }
                }
                buffer += SIDE * columns;
            }
            return mineWord;
        }
        for(unsigned int j = 0; j < n; j++, buffer += columns) {
            bool spiked = false;
            if(active) {
                float in[NPSM];
                unsigned int csCount[NCS > 0 ? NCS : 1] = {0};
                #pragma unroll
                for(unsigned int p = 0; p < NPSM; p++) {
                    in[p] = 0.0f;
                    if(p < g.num_psm) {
                        regs.lin[p] = B200_FADD(regs.lin[p], buffer[myCol[p]]);
                        buffer[myCol[p]] = 0.0f;
                    }
                }
                drawCurrentSources<NCS>(L.neuron, g, 0u, local, t0 + first + j, csCount);
                spiked = neuronCompute(L.neuron, g, 0u, local, t0 + first + j, B200_FMUL((float)(t0 + first + j), L.neuron.dt), regs, in, csCount);
            }
            const unsigned int word = __ballot_sync(0xFFFFFFFFu, spiked);
            if(lane == j) mineWord = word;
        }
        return mineWord;
    };
    // ---- what becomes of the ballots: lane j has that of step first + j, entry number `entry` + j of message `message`
    auto keep = [&](unsigned int word, unsigned int first, unsigned int n, bool send, unsigned int message, unsigned int entry) {
        if(lane < n) {
            words[((first + lane) % W.ring) * RESIDENT_UNITS + warp] = word;
            const b200_neuron_group &g = groups[group];
            // (a recording of fewer steps than these keeps the last ones: no two lanes write the same word)
            if(lane + L.neuron.num_recording_timesteps >= n && L.neuron.num_recording_timesteps && g.record_spk) {
                const unsigned int at = (unsigned int)(((unsigned long long)recAt + first + lane) % L.neuron.num_recording_timesteps);
                g.record_spk[(size_t)at * ((g.num_update + 31u) / 32u) + (local - lane) / 32u] = word;
            }
        }
        const unsigned int mineCount = (lane < n) ? __popc(word) : 0u;
        spikes += mineCount;
        if(!send || !(what & RESIDENT_IS_SOURCE) || !__any_sync(0xFFFFFFFFu, mineCount)) return;
        unsigned int upTo = mineCount;
        #pragma unroll
        for(unsigned int o = 1; o < 32u; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, upTo, o);
            if(lane >= o) upTo += v;
        }
        unsigned int base = 0;
        if(lane == 31u) base = atomicAdd(&sh.sent[message & 1u], upTo);
        base = __shfl_sync(0xFFFFFFFFu, base, 31);
        unsigned short *const body = W.bodies + ((size_t)(message % W.buffers) * G + me) * W.body;
        unsigned int at = base + (upTo - mineCount);
        if(lane < n) {
            const unsigned int row = runTable[group].row;
            for(unsigned int left = word; left; left &= left - 1u, at++) {
                const unsigned int who = __ffs(left) - 1u;
                const unsigned short e = (unsigned short)(((entry + lane) << 10) | (warp << 5) | who);
                if(at < RESIDENT_WINDOW_INLINE) sh.first[message & 1u][at] = e;
                body[at] = e;
                // its runs, while the message is on its way (lengths are multiples of four entries)
                if(L.prefetch) prefetchL2(L.entries + residentTable<const unsigned long long>(L.at.rows)[group] + (size_t)(local - lane + who) * row, row * (unsigned int)sizeof(uint2));
            }
        }
    };
    // the CTA's message, by its last warp, behind a barrier behind the entries: a copy for every RESIDENT_READERS readers (resident.h).
    // Few entries travel with the head, which says of itself when it is there; more lie in the body, behind a fence (all in the body:
    // 0.04 us a step longer with 1000 -> 10 000 neurons, 0.25 with 100 000).
    auto send = [&](unsigned int message) {
        if(warp != warps - 1u) return;
        const unsigned int n = sh.sent[message & 1u], at = (me % readers) * perReader + me / readers;
        const unsigned short *const e = sh.first[message & 1u];
        const unsigned long long tag = tagOf(message);
        if(n > RESIDENT_WINDOW_INLINE) fenceGpu();
        if(lane < L.copies) {
            storeRelaxedGpu(W.heads + ((size_t)(message % W.buffers) * L.copies + lane) * RESIDENT_HEADS + at, (tag << 20) | n,
                            ((unsigned long long)shortTagOf(message) << 48) | ((unsigned long long)e[2] << 32) | ((unsigned long long)e[1] << 16) | e[0]);
        }
        __syncwarp();
        if(lane == 0u) sh.sent[message & 1u] = 0u;
    };
    auto append = [&](unsigned int w, unsigned int j, unsigned int spike) {
        const unsigned int at = atomicAdd(&sh.count[w & 1u][j], 1u);
        if(at < W.cap) list[j * W.cap + at] = spike;
        else atomicOr(&sh.stop, 4u);
    };
    // All CTAs' messages of a number: a reading warp takes every `readers`-th sender, whose heads lie side by side.  Of their
    // entries those for the first `steps` steps of window `to` (the last window of a launch may be short: the others arrive in the next
    // launch, which finds them in the spike lists).
    auto receive = [&](unsigned int message, unsigned int to, unsigned int steps) {
        if(warp < firstReader) return;
        const unsigned int reader = warp - firstReader, sender = lane * readers + reader;
        unsigned int total = 0;
        unsigned long long first = 0;
        if(lane < perReader && sender < G) {
            const ulonglong2 *p = W.heads + ((size_t)(message % W.buffers) * L.copies + me % L.copies) * RESIDENT_HEADS + reader * perReader + lane;
            const unsigned long long tag = tagOf(message);
            unsigned int polls = 0;
            for(;;) {
                const ulonglong2 v = loadRelaxedGpu(p);
                if((v.x >> 20) == tag && (v.y >> 48) == shortTagOf(message)) {
                    total = min((unsigned int)(v.x & 0xFFFFFull), W.body);
                    first = v.y;
                    break;
                }
                if(gaveUp(polls)) break;
            }
        }
        // (entries that did not fit a head are read by other lanes than the one that saw it: __syncwarp() orders the lanes' memory
        // accesses, the vote alone is not said to)
        __syncwarp();
        if(__any_sync(0xFFFFFFFFu, total > RESIDENT_WINDOW_INLINE)) fenceGpu();
        if(steps == 0u) return;
        auto spikeOf = [&](unsigned int e, unsigned int from) { return unitFirst[min(((e >> 5) & 31u) * G + from, L.num_units - 1u)] + (e & 31u); };
        // entries that came with the heads: a lane its sender's
        #pragma unroll
        for(unsigned int u = 0; u < RESIDENT_WINDOW_INLINE; u++) {
            const unsigned int e = (unsigned int)(first >> (16u * u)) & 0xFFFFu;
            if(u < total && total <= RESIDENT_WINDOW_INLINE && (e >> 10) < steps) append(to, e >> 10, spikeOf(e, sender));
        }
        const unsigned short *const bodies = W.bodies + (size_t)(message % W.buffers) * G * W.body;
        for(unsigned int left = __ballot_sync(0xFFFFFFFFu, total > RESIDENT_WINDOW_INLINE); left;) {
            // (loads, places and stores of several senders side by side: one after another each takes its latency)
            constexpr unsigned int SIDE = 4;
            unsigned int from[SIDE], n[SIDE], e[SIDE], at[SIDE];
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) {
                const unsigned int who = left ? __ffs(left) - 1u : 0u;
                n[u] = left ? __shfl_sync(0xFFFFFFFFu, total, who) : 0u;
                left &= left - 1u;
                from[u] = who * readers + reader;
                e[u] = (lane < n[u]) ? __ldcg(bodies + (size_t)from[u] * W.body + lane) : 0xFFFFu;
            }
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) at[u] = ((e[u] >> 10) < steps) ? atomicAdd(&sh.count[to & 1u][e[u] >> 10], 1u) : 0u;
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) {
                if((e[u] >> 10) >= steps) continue;
                if(at[u] < W.cap) list[(e[u] >> 10) * W.cap + at[u]] = spikeOf(e[u], from[u]);
                else atomicOr(&sh.stop, 4u);
            }
            #pragma unroll
            for(unsigned int u = 0; u < SIDE; u++) {
                for(unsigned int i = lane + 32u; i < n[u]; i += 32u) {
                    const unsigned int entry = __ldcg(bodies + (size_t)from[u] * W.body + i);
                    if((entry >> 10) < steps) append(to, entry >> 10, spikeOf(entry, from[u]));
                }
            }
            __syncwarp();
        }
    };
    // spikes from before this launch that arrive in the first n steps of window w
    auto before = [&](unsigned int w, unsigned int n) {
        if(warp < firstReader) return;
        for(unsigned int j = 0; j < n && w * K + j <= delay; j++) {
            for(unsigned int gi = 0; gi < numGroups; gi++) {
                if(!((L.sources[0] >> gi) & 1ull)) continue;
                const b200_neuron_group &g = groups[gi];
                const unsigned int slots = g.num_delay_slots, slot = ringSlot(sh.phase + w * K + j + slots - delay, slots);
                const unsigned int m = min(__ldcg(&g.spk_cnt[slot]), g.num_neurons);
                for(unsigned int i = threadIdx.x - firstReader * 32u; i < m; i += readers * 32u) {
                    const unsigned int id = __ldcg(&g.spk[(size_t)slot * g.num_neurons + i]);
                    if(id < g.num_neurons) append(w, j, (gi << 24) | id);
                    else atomicOr(&state->error, ERR_IND_RANGE);
                }
            }
        }
    };
    // FEED: the steps whose spikes arrive in window w
    unsigned int emitted = 0;
    auto sourceWindow = [&](unsigned int w) {
        if(!ahead) return;
        const int from = (int)(w * K) - 1 - (int)delay;
        const unsigned int first = (unsigned int)max(from, 0), end = (unsigned int)max(min(from + (int)K, (int)L.num_steps), (int)first);
        keep(freeSteps(first, end - first), first, end - first, true, w, (unsigned int)((int)first - from));
        emitted = end;
    };

    if(W.feed) {
        sourceWindow(0u);
        __syncthreads();
        send(0u);
        receive(0u, 0u, min(K, L.num_steps));
        before(0u, min(K, L.num_steps));
        if(K < L.num_steps) sourceWindow(1u);
    }
    unsigned int T = 0, w = 0;
    for(;; T += K, w++) {
        const unsigned int steps = sh.steps;
        if(T >= steps) break;
        const unsigned int n = min(K, steps - T);
        __syncthreads();
        if(W.feed) {
            if(T + K < steps) send(w + 1u);
        }
        else {
            if(w) send(w - 1u);
            if(w >= W.lag) receive(w - W.lag, w, n);
            before(w, n);
            __syncthreads();
        }
        if(const unsigned int stop = sh.stop) {
            if(stop & 1u) return;
            // (LATE, with `may_leave`, only: everything up to here is done)
            sh.steps = T;
            break;
        }
        // ---------------- deliveries ------------------------------------------------------------------
        const unsigned int mineCount = sh.count[w & 1u][lane];
        unsigned int upTo = mineCount;
        #pragma unroll
        for(unsigned int o = 1; o < 32u; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, upTo, o);
            if(lane >= o) upTo += v;
        }
        const unsigned int all = __shfl_sync(0xFFFFFFFFu, upTo, 31);
        if(threadIdx.x == 0) {
            // the account of resident.h ("Busy networks"), window by window
            const long long debt = max((long long)sh.debt + (long long)all * L.weight[0] - (long long)n * L.spare, 0ll);
            sh.debt = (int)min(debt, (long long)RESIDENT_MOST_DEBT);
            // FEED: the populations ahead have got that far
            if(L.may_leave && sh.debt > (int)L.patience) sh.steps = min(steps, T + (W.feed ? 2u * K : K));
        }
        if(const unsigned int parts = W.run_groups) {
            // an item: 32 entries of a run, one load of a lane; eight of them in flight
            constexpr unsigned int SIDE = 8;
            const unsigned int items = all * parts;
            for(unsigned int it = warp; it < items; it += SIDE * warps) {
                uint2 e[SIDE];
                unsigned int buffer[SIDE];
                #pragma unroll
                for(unsigned int u = 0; u < SIDE; u++) {
                    e[u] = make_uint2(RESIDENT_PAD, 0u);
                    buffer[u] = 0u;
                    const unsigned int item = it + u * warps;
                    if(item >= items) continue;
                    const unsigned int s = (parts == 1u) ? item : item / parts;
                    const unsigned int j = __popc(__ballot_sync(0xFFFFFFFFu, s >= upTo));
                    const unsigned int spike = list[j * W.cap + s - __shfl_sync(0xFFFFFFFFu, upTo - mineCount, j)];
                    const ResidentRun run = runTable[spike >> 24];
                    const unsigned int i = (item - s * parts) * 32u + lane;
                    if(i < run.length) e[u] = __ldg(L.entries + run.base() + run.near() + (unsigned long long)(spike & 0xFFFFFFu) * run.row + i);
                    buffer[u] = j * columns;
                }
                #pragma unroll
                for(unsigned int u = 0; u < SIDE; u++) {
                    if(e[u].x == RESIDENT_PAD) continue;
                    residentAdd(acc + buffer[u] + (e[u].x & 0xFFFFu), __uint_as_float(e[u].y));
                    events++;
                }
            }
        }
        const bool mixed = (L.sources[0] & (L.sources[0] - 1ull)) != 0ull;
        for(unsigned int q = 0; q < L.num_spans && all; q++) {
            const ResidentSpan &S = residentTable<const ResidentSpan>(L.at.spans)[q];
            const unsigned int w0 = sh.firstWarp[S.trg_group], targets = sh.firstWarp[S.trg_group + 1] - w0;
            if(!targets) continue;
            // (few units and steps: several warps share a step's spikes)
            const unsigned int parts = (2u * warps - 1u) / (targets * n) + 1u, least = S.gp ? 32u : 16u;
            for(unsigned int it = warp; it < targets * n * parts; it += warps) {
                const unsigned int j = it % n, rest = it / n, part = rest / targets, unitWarp = w0 + rest % targets;
                const unsigned int m = __shfl_sync(0xFFFFFFFFu, mineCount, j), per = ((m + parts - 1u) / parts + least - 1u) / least * least;
                if(part * per >= m) continue;
                const unsigned int unit = unitWarp * G + me - residentTable<const unsigned int>(L.at.unit_start)[S.trg_group];
                const float sum = windowSpan(S, list + j * W.cap, part * per, min(m, (part + 1u) * per), unit, mixed, events);
                const unsigned int col = residentTable<const unsigned int>(L.at.columns)[unitWarp * B200_MAX_PSM + S.psm] & 0xFFFFu;
                if(sum != 0.0f) residentAdd(acc + j * columns + col + lane, sum);
            }
        }
        if(L.count_events && (events >> 24)) {
            atomicAdd(&state->synaptic_events, (unsigned long long)events);
            events = 0u;
        }
        if(threadIdx.x < 32u) sh.count[(w + 1u) & 1u][threadIdx.x] = 0u;
        __syncthreads();
        // ---------------- neuron updates, and what the next window needs ----------------------------------
        if(W.feed) {
            const unsigned int end = sh.steps;
            if(T + K < end) {
                receive(w + 1u, w + 1u, min(K, end - T - K));
                before(w + 1u, min(K, end - T - K));
            }
            if(T + 2u * K < end) sourceWindow(w + 2u);
        }
        if(mine && !ahead) {
            const bool source = !W.feed;
            if(what & (RESIDENT_IS_POISSON | RESIDENT_IS_ARRAY)) keep(freeSteps(T, n), T, n, source, w, 0u);
            else keep(fedSteps(T, n), T, n, source, w, 0u);
        }
    }
    // ---------------- what the launch leaves in memory ----------------------------------------------------
    // (populations ahead have not got to the end yet: the spikes they still have arrive in the next launch)
    const unsigned int step = sh.steps;
    if(ahead) {
        for(; emitted < step; emitted += min(K, step - emitted)) {
            const unsigned int n = min(K, step - emitted);
            keep(freeSteps(emitted, n), emitted, n, false, 0u, 0u);
        }
    }
    __syncthreads();
    // one more message from everybody: nobody reads the spike lists any more.  (w: windows done; LATE: the last one's spikes have
    // not been sent, unless it could not be done)
    const unsigned int last = (W.feed || sh.stop) ? w : w - 1u;
    send(last);
    receive(last, 0u, 0u);
    __syncthreads();
    if(sh.stop & 1u) return;
    const unsigned long long doneNow = sh.done + step;
    const unsigned int k = (sh.phase + step) % sh.period, period = sh.period;
    // lists of the last steps: emptied by the first CTA (and the one the next step writes), filled by all
    const unsigned int lists = min(L.history, step);
    if(me == 0) {
        for(unsigned int i = threadIdx.x; i < numGroups * (lists + 1u); i += blockDim.x) {
            const b200_neuron_group &g = groups[i % numGroups];
            const unsigned int t = i / numGroups;      // 0: the next step, t: t - 1 steps ago
            if(t < g.num_delay_slots) g.spk_cnt[ringSlot(k + 1u + g.num_delay_slots - t, g.num_delay_slots)] = 0u;
        }
        __threadfence();
        __syncthreads();
        if(threadIdx.x == 0) storeRelaxedGpu(L.leave, L.launch);
    }
    else {
        if(threadIdx.x == 0) {
            unsigned int polls = 0;
            while(loadRelaxedGpu(L.leave) != L.launch && !gaveUp(polls)) {}
            __threadfence();
        }
        __syncthreads();
    }
    if(mine) {
        const b200_neuron_group &g = groups[group];
        for(unsigned int t = 0; t < lists && t + 1u < g.num_delay_slots; t++) {
            const unsigned int b = words[((step - 1u - t) % W.ring) * RESIDENT_UNITS + warp];
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
        if(active) storeNeuron(g, local, regs, false);
    }
    if(L.count_events) {
        // (halves, so that the sum over a warp does not pass 32 bits)
        const unsigned long long e = __reduce_add_sync(0xFFFFFFFFu, events & 0xFFFFu) + ((unsigned long long)__reduce_add_sync(0xFFFFFFFFu, events >> 16) << 16);
        const unsigned int s = __reduce_add_sync(0xFFFFFFFFu, spikes);
        if(lane == 0 && e) atomicAdd(&state->synaptic_events, e);
        if(lane == 0 && s) atomicAdd(&state->spikes, (unsigned long long)s);
    }
    // (every CTA has sent its last message, so every CTA has read the counters)
    if(me == 0 && threadIdx.x == 0) {
        state->timestep = t0 + step;
        state->steps_done = doneNow;
        state->phase = k;
        residentSettle(L, *state, sh.debt, step, doneNow);
    }
}
}   // namespace b200
