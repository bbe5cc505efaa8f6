// k_u1.cu -- small builds: the merged launch of the low-register classes (unit.cuh).
#include "unit.cuh"

namespace liberi {
template cudaError_t launch_unit_t<true, double>(const UnitArgs &, int, cudaStream_t);
template cudaError_t launch_unit_t<true, float>(const UnitArgs &, int, cudaStream_t);
}  // namespace liberi
