// se2gpu_internal.h -- the solver handle's layout and the helpers that the
// single-shot API (se2gpu_api.cu) shares with the batched ensemble
// (se2gpu_ensemble.cu).  Not part of the public interface.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "se2gpu.h"
#include "se2gpu_persist_params.h"

// a tile configuration of the FP32 modes, set up on a handle
struct se2gpu_tiles {
  CUtensorMap maps[2][6];        // per input buffer set: region u, cu, owned w, cw; cell constants, 1/M
  int4 *bounds;                  // per tile: source and receiver list bounds
  int4 *src, *rec;               // per-tile list entries
  size_t first, src_at, rec_at;  // their places: bounds in the handle's table (tiles.bounds is its start), the lists from bounds
  int config, ntx, nty, grid;
  bool halo;                     // else its step keeps element forces (se2gpu_f32ef.cuh, se2gpu_f32df.cuh)
};

struct se2gpu_solver {
  int pageable;      // the device reads and writes pageable host memory (cudaDevAttrPageableMemoryAccess)
  int mx, my, p, n1, npe, nx_g, ny_g, precision;
  long nnodes;
  int nsrc, nrec, trace_cap, rows_written;
  bool pending_record;
  double dt;
  int device, nsm;
  cudaStream_t stream, own_stream;
  size_t tsize;                  // compute precision (4 or 8 bytes)
  // FP64 state: two buffer sets of packed u, v; a of the last step (f64[0][0] the allocation of all); element forces of a step
  // (FP32 steps without a halo too: 8 bytes per element node, two-float 16; ef[0] is the allocation of both
  // and of 1/M); scaled derivative tables (Dx the allocation of all that follow)
  double2 *f64[2][2], *a64, *ef[2];
  double *rmass, *Dx, *Dy, *f64_consts;
  int2 *src_xy;                  // first node of each source's element
  int cur;
  int unfinished;                // FP64: the begun step without its v and a yet: its row of stf_dev + 1 (0: none)
  // FP32 leapfrog state (padded): u, w, cu, cw per buffer set, a of the last step
  int pitch;
  float2 *pu[2], *pw[2], *pcu[2], *pcw[2], *pa;
  float *pminv, *rbuf[2];
  unsigned long long *mass_bad;  // first node with a mass that is not positive (device check at create)
  cudaEvent_t side_done[2];      // se2gpu_create: set-up work on side streams not yet joined
  int rlast;
  float4 *cellc;                 // plain and Kahan modes: (lam detJ, mu detJ, d xi/dx, d eta/dy) per cell
  se2gpu_tiles tiles, single;    // what blocks run; what a block of one step runs, where that is another (bounds set)
  int config;                    // selected configuration number (tiles.config: the tiles that it stands for)
  int auto_config, auto_tiles;   // the number of the mesh's own choice, and its tiles (se2p::first_config)
  std::vector<int> *src_elem_h, *rec_elem_h;
  int *err_dev;
  // tables in compute precision
  void *mass, *lam, *mu, *J00, *J11, *iJ00, *iJ11, *D, *wq, *src_vals;
  double *Dd, *iJ00d, *iJ11d, *stf_dev, *traces, *norm_part;
  int stf_cap;
  int *rec_node, *rec_elem, *rec_gll;
  void *scratch_u, *scratch_f;   // assemble_linear_form staging (packed)
  long launches;
  char err[512];
};

// se2gpu_create; in_ensemble: the tile configuration that all shots of a degree share, whatever the
// mesh size
int se2gpu_internal_create(const se2gpu_problem *P, int precision, int trace_capacity, bool in_ensemble, se2gpu_solver **out);
// FP32 persistent-kernel parameters of a handle (no per-step pointers set)
se2p::Params se2gpu_internal_f32_params(se2gpu_solver *h);
// set the thread's message returned by se2gpu_last_error(NULL)
void se2gpu_internal_set_error(const char *msg);
