// acfdtd_resident_f32.cu -- the resident sweep in single precision.

#include "acfdtd_resident_kernel.cuh"

namespace acf {

template ResidentPlan resident_plan<float>(int, int, int, int, bool, int, size_t);
template cudaError_t resident_launch<float>(const ResidentPlan &, const ResidentRun<float> &, int64_t, cudaStream_t);

}  // namespace acf
