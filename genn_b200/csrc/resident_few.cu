// Instances of the target-resident kernel (resident.h): several ring depths or axonal delays, blocks of up to 640 threads.
#include "resident_step.cuh"

namespace b200
{
const void *residentFew(int npsm, int ncs) { return residentInstance<false, RESIDENT_FEW>(npsm, ncs); }
}   // namespace b200
