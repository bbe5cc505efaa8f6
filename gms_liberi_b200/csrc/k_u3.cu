// k_u3.cu -- small builds: the merged FP32 launch of the high-register classes (unit.cuh).
#include "unit.cuh"

namespace liberi {
template cudaError_t launch_unit_t<false, float>(const UnitArgs &, int, cudaStream_t);
}  // namespace liberi
