// se2gpu_f32df_launch.h -- tile configurations and launch of the two-float step (se2gpu_f32df.cu).
#pragma once
#include <cuda_runtime.h>

#include "se2gpu_persist_params.h"

namespace se2p {

// Tile configurations of the two-float mode, X(degree, elements per tile edge, threads) for the step
// without a halo (threads >= edge^2 (degree + 1), whole warps) and H(degree, edge, threads) for the
// one that recomputes a halo of elements (se2gpu_persist.cuh).  Per degree the tile for large meshes
// comes first and those for small meshes last: a number kept from a list of other tiles then
// selects one that a large mesh can run on.  The halo is kept where it was faster: large meshes of degrees 2 and 3, whose
// elements are cheap against the node part and the forces' traffic (a million nodes: 75 against 78
// us a step, 69 against 72).  Everywhere else it lost: at 2.5M nodes 257 against 234 us (degree 1),
// 163 / 153 (4), 200 / 160 (5), 219 / 169 (6), 304 / 176 (7), 276 / 196 (8).  Small tiles with
// about a thread per node are for meshes that leave SMs idle, where the step is a chain of latencies:
// more threads shorten the node part (20000 nodes: degree 2 8.6 -> 5.1 us, 3 7.8 -> 5.6, 4 12.2
// -> 7.8, 5 14.2 -> 8.6, 6 14.5 -> 10.2, 7 19.4 -> 11.9, 8 20.0 -> 12.4).
#define SE2P_DF_CONFIGS(X, H)                                                               \
  X(1, 12, 288) X(1, 8, 320) X(1, 6, 192)                                                   \
  H(2, 12, 512) X(2, 8, 192) X(2, 6, 192) X(2, 4, 96)                                       \
  H(3, 7, 256) X(3, 4, 64) X(3, 4, 192)                                                     \
  X(4, 5, 128) X(4, 7, 256) X(4, 6, 192) X(4, 3, 64) X(4, 3, 192) X(4, 2, 96)               \
  X(5, 4, 96) X(5, 6, 224) X(5, 2, 128)                                                     \
  X(6, 6, 256) X(6, 3, 64) X(6, 2, 192)                                                     \
  X(7, 4, 128) X(7, 3, 96) X(7, 2, 256)                                                     \
  X(8, 5, 256) X(8, 3, 96) X(8, 1, 96)

// exchange rows: float4 between rows and between elements
__host__ __device__ constexpr int df_row_pitch(int p) { return (p + 1) | 1; }
__host__ __device__ constexpr int df_elem_pitch(int p) { return (p + 1) * df_row_pitch(p); }

// CTAs per SM the registers are sized for: 28 warps (72 registers) up to degree 5, 12 (the 110 that
// the rolled code takes) above, within the shared memory.  20, 24 and 32 warps at degree 4: 159,
// 157 and 159 against 154 us a step at 2.5M nodes
__host__ __device__ constexpr int df_min_blocks(int p, int te, int nt)
{
  const int rw = te * p + 1;
  const long smem = 16L * ((long)rw * rw + 2L * te * te * df_elem_pitch(p)) + 1024;
  const int by_smem = (int)(233472 / smem), by_regs = (p <= 5 ? 896 : 384) / nt;
  const int n = by_smem < by_regs ? by_smem : by_regs;
  return n < 1 ? 1 : n;
}

struct DfShape {
  int p, te, nt;
  size_t smem;
  const void *fn;
  bool halo;
};

// configuration of degree p, with or without a halo; false: no such configuration
bool df_shape(int p, int config, DfShape *s);
// the step without a halo (the other one: launch_step)
cudaError_t df_launch(int p, int config, const EfParams &q, bool dependent, cudaStream_t st);

}  // namespace se2p
