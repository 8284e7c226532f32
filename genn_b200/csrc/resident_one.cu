// Instances of the target-resident kernel (resident.h): one ring depth and one axonal delay, larger blocks.
#include "resident_step.cuh"

namespace b200
{
const void *residentOne(int npsm, int ncs) { return residentInstance<true, RESIDENT_BLOCK>(npsm, ncs); }
}   // namespace b200
