// se2gpu_launch.h -- launch entry points of the FP32 internal force.
#pragma once
#include <cuda_runtime.h>
#include "se2gpu_kernels.cuh"

namespace se2 {

cudaError_t prepare_f32(int p);  // raise the dynamic shared-memory limit (current device)
cudaError_t launch_force_f32(int p, const ForceParams &prm, cudaStream_t st);

}  // namespace se2
