// se2gpu_f64_launch.h -- launch entry points of the FP64 kernels (se2gpu_f64.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace se2 {

struct F64Params {
  int mx, my, nx_g, ny_g;
  int ntx, ntiles, nsamp;            // tiles, then nsamp CTAs that sample the receivers
  int trigger;                       // let the next launch begin during the divergence
  int mode;                          // F64_START, F64_MIDDLE or F64_FORCE
  const double2 *u_in, *v_in, *a_in; // START: u, v, a; MIDDLE: u', v* of the previous step; FORCE: u
  const double2 *ef_in;              // MIDDLE: the previous step's element forces
  double2 *u_out, *v_out, *ef_out;   // u', v* and element forces of this step
  const double *mass, *rmass;        // M, and 1/M rounded (0 where the division has to be taken)
  const double *lam, *mu, *J00, *J11;
  const double *Dx, *Dy;             // [mx][npe], [my][npe]: dN/dx = (1/J00) D, dN/dy = (1/J11) D
  const double *wq;
  const double *constants;           // {1, -0}
  double c_dt, c_u, c_v;             // dt, 0.5*dt*dt, 0.5*dt (computed on the host as in se2wave.c:4726-4745)
  int nsrc;
  const int2 *src_xy;                // first node (column, row) of each source's element
  const double *src_vals;            // [nsrc][2*npe]
  const double *stf;                 // the previous step's values (MIDDLE and the last pass)
  int nrec;                          // receivers to sample (0: none)
  const int *rec_elem, *rec_gll;
  const double *Dd, *iJ00d, *iJ11d;
  double *trace_row;
};

enum { F64_START = 0, F64_MIDDLE = 1, F64_FORCE = 2 };

struct F64TileShape { int ex, ey, threads; };   // elements along x and y
F64TileShape f64_tile(int p, const F64Params &q, int nsm);   // what f64_launch_step runs on the mesh of q
// one START, MIDDLE or FORCE launch (q.mode); fills in the tile grid
cudaError_t f64_launch_step(int p, const F64Params &q, int nsm, cudaStream_t st);
// v and a of the block's last step from the element forces q.ef_in (v in place)
cudaError_t f64_launch_last(int p, const F64Params &q, double2 *v, double2 *a, cudaStream_t st);
// nodal internal force from the element forces q.ef_in
cudaError_t f64_launch_force(int p, const F64Params &q, double2 *f, cudaStream_t st);
// receiver rows of the state (q.u_in, q.v_in, q.a_in)
cudaError_t f64_launch_record(int p, const F64Params &q, cudaStream_t st);
cudaError_t f64_launch_reciprocal(const double *mass, double *r, size_t n, int nsm, cudaStream_t st);

}  // namespace se2
