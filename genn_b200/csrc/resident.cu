// The target-resident time-step path (resident.h): which instance, and the private copy of the synapses.
#include "resident.h"
#include "common.cuh"

namespace b200
{
// one each in resident_one_few.cu, resident_one.cu, resident_few.cu, resident_many.cu
const void *residentOneFew(int npsm, int ncs);
const void *residentOne(int npsm, int ncs);
const void *residentFew(int npsm, int ncs);
const void *residentMany(int npsm, int ncs);

const void *residentKernelFor(int npsm, int ncs, bool one_class, unsigned int threads)
{
    const bool few = threads <= RESIDENT_FEW;
    if(one_class) return few ? residentOneFew(npsm, ncs) : residentOne(npsm, ncs);
    return few ? residentFew(npsm, ncs) : residentMany(npsm, ncs);
}

// ---- building the runs ---------------------------------------------------------------------------
// One CTA per source neuron: counts (pass 0) or places (pass 1) its synapses by the CTA that holds the target.
__global__ void __launch_bounds__(256)
residentBuildKernel(const ResidentBuild B, int pass, unsigned int *longest, const ResidentRun *runs, uint2 *entries, StepState *state)
{
    __shared__ unsigned int cursor[2 * RESIDENT_MAX_CTAS];      // per CTA: behind the head, and of the head
    unsigned long long synapses = 0;
    for(unsigned int pre = blockIdx.x; pre < B.num_src; pre += gridDim.x) {
        for(unsigned int c = threadIdx.x; c < 2u * RESIDENT_MAX_CTAS; c += blockDim.x) cursor[c] = 0u;
        __syncthreads();
        for(unsigned int gi = 0; gi < B.num_groups; gi++) {
            const b200_synapse_group &g = B.groups[gi];
            const unsigned int len = min(g.row_length[pre], g.row_stride);
            synapses += len;
            const unsigned int trg = B.target[gi] >> 8, psm = B.target[gi] & 0xFFu;
            const unsigned int firstUnit = B.unit_start[trg];
            const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
            for(unsigned int j = threadIdx.x; j < len; j += blockDim.x) {
                const unsigned long long s = (unsigned long long)pre * g.row_stride + j;
                const unsigned int post = (g.ind_bytes == 1) ? static_cast<const uint8_t*>(g.ind)[s]
                    : (g.ind_bytes == 2) ? static_cast<const uint16_t*>(g.ind)[s] : static_cast<const uint32_t*>(g.ind)[s];
                if(post >= g.num_trg) {
                    atomicOr(&state->error, ERR_IND_RANGE);
                    continue;
                }
                const unsigned int unit = firstUnit + (post >> 5), cta = unit % B.grid, w = unit / B.grid;
                unsigned int d = B.late;
                if(g.max_den_delay) d = (unsigned int)g.d[s] % g.max_den_delay;
                const bool near = B.split && d == 0u;
                const unsigned int at = atomicAdd(&cursor[near ? RESIDENT_MAX_CTAS + cta : cta], 1u);
                if(pass == 0) continue;
                const ResidentRun run = runs[(unsigned long long)cta * B.runs_stride];
                if(at >= (near ? run.near() : run.length)) continue;        // (counted in pass 0: only if the arrays changed in between)
                const unsigned int col = B.columns[((unsigned long long)cta * RESIDENT_UNITS + w) * B200_MAX_PSM + psm];
                const unsigned int cls = col >> 16, c = (col & 0xFFFFu) + (post & 31u), weight = __float_as_uint(constant ? g.wu_params[0] : g.g[s]);
                entries[run.base() + (near ? 0u : run.near()) + (unsigned long long)pre * run.row + at] = make_uint2((cls << 30) | (d << 16) | c, weight);
            }
        }
        __syncthreads();
        if(pass == 0) {
            for(unsigned int c = threadIdx.x; c < B.grid; c += blockDim.x) {
                unsigned int *cell = &longest[(unsigned long long)c * B.runs_stride];
                if(cursor[c] > *cell) atomicMax(cell, cursor[c]);
                if(cursor[RESIDENT_MAX_CTAS + c] > *B.near_longest) atomicMax(B.near_longest, cursor[RESIDENT_MAX_CTAS + c]);
            }
        }
        __syncthreads();
    }
    if(pass == 0 && threadIdx.x == 0 && synapses) atomicAdd(B.synapses, synapses);
}

cudaError_t residentBuild(const ResidentBuild &B, int pass, unsigned int *longest, const ResidentRun *runs, uint2 *entries, StepState *state,
                          unsigned int blocks, cudaStream_t stream)
{
    residentBuildKernel<<<blocks, 256, 0, stream>>>(B, pass, longest, runs, entries, state);
    return cudaPeekAtLastError();
}
}   // namespace b200
