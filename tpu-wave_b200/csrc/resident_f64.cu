// On-chip runs of the elastic step (resident.cuh) for FP64 fields.
#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<double, RES_ELASTIC>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<double, RES_ELASTIC>(const ResArgs<double> &, int, bool, const ResPlan &, cudaStream_t);
}  // namespace tw
