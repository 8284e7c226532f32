// Instances of the target-resident kernel (resident.h): several ring depths or axonal delays, larger blocks.
#include "resident_step.cuh"

namespace b200
{
const void *residentMany(int npsm, int ncs) { return residentInstance<false, RESIDENT_BLOCK>(npsm, ncs); }
}   // namespace b200
