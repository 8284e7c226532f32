// Instances of the target-resident kernel (resident.h): one ring depth and one axonal delay, blocks of up to 640 threads.
#include "resident_step.cuh"

namespace b200
{
const void *residentOneFew(int npsm, int ncs) { return residentInstance<true, RESIDENT_FEW>(npsm, ncs); }
}   // namespace b200
