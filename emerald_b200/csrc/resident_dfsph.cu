// The resident solve of one method (its own source file, so that the methods
// compile in parallel).
#include "resident_solve.cuh"

namespace emerald {

template bool resident_limits_of<kDfsph>(bool, ResidentLimits&);
template uint32_t resident_smem_of<kDfsph>(uint32_t, uint32_t);
template cudaError_t launch_resident_of<kDfsph>(Arena const&, ResidentPlan const&, bool, bool,
                                            cudaStream_t);

}  // namespace emerald
