// acfdtd_resident_f64.cu -- the resident sweep in double precision.

#include "acfdtd_resident_kernel.cuh"

namespace acf {

template ResidentPlan resident_plan<double>(int, int, int, int, bool, int, size_t);
template cudaError_t resident_launch<double>(const ResidentPlan &, const ResidentRun<double> &, int64_t, cudaStream_t);

}  // namespace acf
