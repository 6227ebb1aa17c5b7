// On-chip runs of the acoustic step (resident.cuh) for FP32 fields.
#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<float, RES_AC_FREE>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_AC_FREE>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);
template cudaError_t prepare_resident<float, RES_AC_PER>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_AC_PER>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);
}  // namespace tw
