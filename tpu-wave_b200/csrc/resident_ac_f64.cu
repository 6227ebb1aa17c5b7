// On-chip runs of the acoustic step (resident.cuh) for FP64 fields.
#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<double, RES_AC_FREE>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<double, RES_AC_FREE>(const ResArgs<double> &, int, bool, const ResPlan &, cudaStream_t);
template cudaError_t prepare_resident<double, RES_AC_PER>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<double, RES_AC_PER>(const ResArgs<double> &, int, bool, const ResPlan &, cudaStream_t);
template cudaError_t prepare_resident_shots<double, RES_AC_FREE>(int, bool, int);
template cudaError_t launch_resident_shots<double, RES_AC_FREE>(const ResArgs<double> *, const int *, int, int, size_t, int, bool, cudaStream_t);
template cudaError_t prepare_resident_shots<double, RES_AC_PER>(int, bool, int);
template cudaError_t launch_resident_shots<double, RES_AC_PER>(const ResArgs<double> *, const int *, int, int, size_t, int, bool, cudaStream_t);
}  // namespace tw
