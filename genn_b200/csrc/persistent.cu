// Instances of the persistent time-step kernels that share their input buffers between CTAs (fused_step.cuh,
// stream_step.cuh), by the largest number of postsynaptic models and current sources of any neuron group.
#include "fused_step.cuh"
#include "stream_step.cuh"

namespace b200
{
#define B200_SHAPES(USE) USE(1, 0); USE(1, 1); USE(1, B200_MAX_CS); USE(2, 0); USE(2, 1); USE(2, B200_MAX_CS); \
    USE(B200_MAX_PSM, 0); USE(B200_MAX_PSM, 1); USE(B200_MAX_PSM, B200_MAX_CS)

const void *fusedKernelFor(int npsm, int ncs)
{
#define B200_USE(P, C) if(npsm == P && ncs == C) return (const void*)fusedStepKernel<P, C>
    B200_SHAPES(B200_USE);
#undef B200_USE
    return nullptr;
}

const void *streamKernelFor(int npsm, int ncs, bool sharded)
{
#define B200_USE(P, C) if(npsm == P && ncs == C) return sharded ? (const void*)streamStepKernel<P, C, true> : (const void*)streamStepKernel<P, C, false>
    B200_SHAPES(B200_USE);
#undef B200_USE
    return nullptr;
}
}   // namespace b200
