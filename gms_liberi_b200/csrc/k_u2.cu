// k_u2.cu -- small builds: the merged FP64 launch of the high-register classes (unit.cuh).
#include "unit.cuh"

namespace liberi {
template cudaError_t launch_unit_t<false, double>(const UnitArgs &, int, cudaStream_t);
}  // namespace liberi
