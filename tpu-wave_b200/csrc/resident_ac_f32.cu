// On-chip runs of the acoustic step (resident.cuh) for FP32 fields.
#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<float, RES_AC_FREE>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_AC_FREE>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);
template cudaError_t prepare_resident<float, RES_AC_PER>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_AC_PER>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);
template cudaError_t prepare_resident_shots<float, RES_AC_FREE>(int, bool, int);
template cudaError_t launch_resident_shots<float, RES_AC_FREE>(const ResArgs<float> *, const int *, int, int, size_t, int, bool, cudaStream_t);
template cudaError_t prepare_resident_shots<float, RES_AC_PER>(int, bool, int);
template cudaError_t launch_resident_shots<float, RES_AC_PER>(const ResArgs<float> *, const int *, int, int, size_t, int, bool, cudaStream_t);
}  // namespace tw
