// The resident solve of one method (its own source file, so that the methods
// compile in parallel).
#include "resident_solve.cuh"

namespace emerald {

template bool resident_limits_of<kIisph>(bool, ResidentLimits&);
template uint32_t resident_smem_of<kIisph>(uint32_t, uint32_t);
template cudaError_t launch_resident_of<kIisph>(Arena const&, ResidentPlan const&, bool, bool,
                                            cudaStream_t);

}  // namespace emerald
