// se2gpu_f32.cu -- the internal force in plain FP32, degrees 1..8: the entry point
// se2gpu_assemble_linear_form[_device] on an FP32 handle.  FP32 time stepping runs the
// kernels of se2gpu_f32p.cu, se2gpu_f32ef.cu and se2gpu_f32df.cu.
#include "se2gpu_launch.h"

namespace se2 {

template <int P>
static cudaError_t prep()
{
  return cudaFuncSetAttribute(force_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_layout<P>().total);
}

template <int P>
static cudaError_t launch(const ForceParams &prm, cudaStream_t st)
{
  ForceParams q = prm;
  q.ntx = (q.mx + Tile<P>::TE - 1) / Tile<P>::TE;
  q.nty = (q.my + Tile<P>::TE - 1) / Tile<P>::TE;
  force_kernel<P><<<q.ntx * q.nty, 256, smem_layout<P>().total, st>>>(q);
  return cudaGetLastError();
}

#define SE2_DISPATCH(fn, ...)                                               \
  switch (p) {                                                              \
    case 1: return fn<1>(__VA_ARGS__); case 2: return fn<2>(__VA_ARGS__);   \
    case 3: return fn<3>(__VA_ARGS__); case 4: return fn<4>(__VA_ARGS__);   \
    case 5: return fn<5>(__VA_ARGS__); case 6: return fn<6>(__VA_ARGS__);   \
    case 7: return fn<7>(__VA_ARGS__); case 8: return fn<8>(__VA_ARGS__);   \
    default: break;                                                         \
  }

cudaError_t prepare_f32(int p) { SE2_DISPATCH(prep) return cudaErrorInvalidValue; }
cudaError_t launch_force_f32(int p, const ForceParams &prm, cudaStream_t st)
{
  SE2_DISPATCH(launch, prm, st)
  return cudaErrorInvalidValue;
}

}  // namespace se2
