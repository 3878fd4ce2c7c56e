// Explicit instantiation of the table half-sweep's launchers.
#include "sweep_table.cuh"

namespace ginf_gpu {
template cudaError_t launch_table<float, float>(const RecordFormat &, const SweepParams &, cudaStream_t, int);
template cudaError_t launch_table<float, __half>(const RecordFormat &, const SweepParams &, cudaStream_t, int);
template cudaError_t launch_table<int, int>(const RecordFormat &, const SweepParams &, cudaStream_t, int);
}  // namespace ginf_gpu
