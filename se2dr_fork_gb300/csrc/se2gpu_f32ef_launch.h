// se2gpu_f32ef_launch.h -- tile configurations and launch of the plain and Kahan step without a halo
// (se2gpu_f32ef.cu).
#pragma once
#include <cuda_runtime.h>

#include "se2gpu_persist_params.h"

namespace se2p {

// Tile configurations, X(degree, elements per tile edge, threads >= edge^2 (degree + 1)), which follow
// those of SE2P_CONFIGS in a handle's numbering: tiles with about a thread per node, for meshes that
// leave SMs idle.
#define SE2P_EF_CONFIGS(X)                                                                  \
  X(1, 8, 320) X(2, 6, 192) X(3, 4, 192) X(4, 3, 192) X(5, 2, 128) X(6, 2, 192) X(7, 2, 256) X(8, 1, 96)

// shared memory: exchange rows, displacement (and its Kahan terms)
constexpr size_t ef_smem(int p, int te, bool kahan, int xs)
{
  return 8 * ((size_t)2 * te * te * xs + (size_t)(te * p + 1) * (te * p + 1) * (kahan ? 2 : 1));
}
// CTAs per SM the registers are sized for: 32 warps up to degree 5, 24 above (no spills)
constexpr int ef_min_blocks(int p, int nt) { return (p <= 5 ? 1024 : 768) / nt; }

struct EfShape {
  int p, te, nt;
  size_t smem[2];       // [kahan]
  const void *fn[2];    // ef_step<...> [kahan]
};

cudaError_t ef_set_tables(int p, const double *D, const double *w1d);
bool ef_shape(int p, int k, EfShape *s);   // the k-th of degree p; false: no such configuration
cudaError_t ef_launch(int p, int k, bool kahan, const EfParams &q, bool dependent, cudaStream_t st);

}  // namespace se2p
