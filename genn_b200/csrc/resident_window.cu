// Instances of the target-resident kernel that exchanges spikes once for a window of steps (resident_window.cuh).
#include "resident_window.cuh"

namespace b200
{
const void *residentWindowKernelFor(int npsm, int ncs)
{
#define B200_WINDOW(P, C) if(npsm == P && ncs == C) return (const void*)residentWindowKernel<P, C>
    B200_WINDOW(1, 0); B200_WINDOW(1, 1); B200_WINDOW(1, B200_MAX_CS);
    B200_WINDOW(2, 0); B200_WINDOW(2, 1); B200_WINDOW(2, B200_MAX_CS);
    B200_WINDOW(B200_MAX_PSM, 0); B200_WINDOW(B200_MAX_PSM, 1); B200_WINDOW(B200_MAX_PSM, B200_MAX_CS);
#undef B200_WINDOW
    return nullptr;
}
}   // namespace b200
