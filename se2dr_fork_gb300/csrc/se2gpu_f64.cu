// se2gpu_f64.cu -- FP64 (reference operation order) kernels, degrees 1..8, and their launches.
#include <algorithm>

#include "se2gpu_f64_launch.h"
#include "se2gpu_f64.cuh"

namespace se2 {

#define SE2_DISPATCH(fn, ...)                                               \
  switch (p) {                                                              \
    case 1: return fn<1>(__VA_ARGS__); case 2: return fn<2>(__VA_ARGS__);   \
    case 3: return fn<3>(__VA_ARGS__); case 4: return fn<4>(__VA_ARGS__);   \
    case 5: return fn<5>(__VA_ARGS__); case 6: return fn<6>(__VA_ARGS__);   \
    case 7: return fn<7>(__VA_ARGS__); case 8: return fn<8>(__VA_ARGS__);   \
    default: return {};                                                     \
  }

template <class A> struct arg { typedef A type; };   // (keeps A out of the deduction)
// launch, beginning while the launch before it in the stream drains
template <class... A>
static cudaError_t launch_dependent(void (*fn)(A...), dim3 grid, int threads, cudaStream_t st, typename arg<A>::type... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

template <int P, int SIZE>
static long tiles(const F64Params &q)
{
  typedef F64Tile<P, SIZE> T;
  return (long)((q.mx + T::TX - 1) / T::TX) * ((q.my + T::TY - 1) / T::TY);
}

// FP64 warp instructions of the busiest SM: a tile's element points (20 (p+1) each, strain
// and divergence) and its nodes (about 40 each), in whole warps
template <int P, int SIZE>
static long cost(const F64Params &q, int nsm)
{
  typedef F64Tile<P, SIZE> T;
  const long points = (T::TX * T::TY * (P + 1) * (P + 1) + 31) / 32;
  const long nodes = ((T::TX * P + 1) * (T::TY * P + 1) + 31) / 32;
  return ((tiles<P, SIZE>(q) + nsm - 1) / nsm) * (points * 20 * (P + 1) + nodes * 40);
}

template <int P, int SIZE>
static cudaError_t step_t(F64Params &q, int nsm, cudaStream_t st)
{
  typedef F64Tile<P, SIZE> T;
  q.ntx = (q.mx + T::TX - 1) / T::TX;
  q.ntiles = (int)tiles<P, SIZE>(q);
  const int per = T::NT / 32;   // receivers per sampling CTA and pass
  q.nsamp = std::min((q.nrec + per - 1) / per, 256);
  // A launch made while the one before it drains starts about 2 us sooner (100-step blocks:
  // 9.9 -> 7.3 us per step at 300 nodes, 27.6 -> 25.8 at 60000).  Letting it begin before
  // that one's last CTAs have ended gains another 0.5-1 us where every SM has at most one
  // tile; with more, the early CTAs fill the SMs that are idle at that moment and
  // unbalance the rest (13.5 -> 24 us at degree 4, 35 x 35 elements).
  q.trigger = q.ntiles <= nsm;
  if (q.mode == F64_MIDDLE) return launch_dependent(f64_step<P, SIZE>, dim3(q.ntiles + q.nsamp), T::NT, st, q);
  f64_step<P, SIZE><<<q.ntiles + q.nsamp, T::NT, 0, st>>>(q);
  return cudaGetLastError();
}

// The tile size with the least work on the busiest SM.  Over all degrees and 300 to 400000
// nodes this is within 1 % (mean) and 11 % (worst) of the best of the three as timed; taking
// always one size costs up to 3.5x (degree 6, 9 x 9 elements: 11.8, 16.1 or 38.1 us).
template <int P>
static int pick(const F64Params &q, int nsm)
{
  const long c0 = cost<P, 0>(q, nsm), c1 = cost<P, 1>(q, nsm), c2 = cost<P, 2>(q, nsm);
  return (c0 < c1 && c0 < c2) ? 0 : (c1 < c2) ? 1 : 2;
}

template <int P>
static cudaError_t step(const F64Params &prm, int nsm, cudaStream_t st)
{
  F64Params q = prm;
  switch (pick<P>(q, nsm)) {
    case 0: return step_t<P, 0>(q, nsm, st);
    case 1: return step_t<P, 1>(q, nsm, st);
    default: return step_t<P, 2>(q, nsm, st);
  }
}

template <int P>
static F64TileShape shape(const F64Params &q, int nsm)
{
  static const F64TileShape t[3] = {{F64Tile<P, 0>::TX, F64Tile<P, 0>::TY, F64Tile<P, 0>::NT},
                                    {F64Tile<P, 1>::TX, F64Tile<P, 1>::TY, F64Tile<P, 1>::NT},
                                    {F64Tile<P, 2>::TX, F64Tile<P, 2>::TY, F64Tile<P, 2>::NT}};
  return t[pick<P>(q, nsm)];
}
F64TileShape f64_tile(int p, const F64Params &q, int nsm) { SE2_DISPATCH(shape, q, nsm) }

static dim3 node_grid(const F64Params &q) { return dim3((q.nx_g + 255) / 256, std::min(q.ny_g, 65535)); }

template <int P>
static cudaError_t last(const F64Params &q, double2 *v, double2 *a, cudaStream_t st)
{
  return launch_dependent(f64_last<P>, node_grid(q), 256, st, q, v, a);
}

template <int P>
static cudaError_t force(const F64Params &q, double2 *f, cudaStream_t st)
{
  return launch_dependent(f64_force<P>, node_grid(q), 256, st, q, f);
}

template <int P>
static cudaError_t record(const F64Params &q, cudaStream_t st)
{
  f64_record<P><<<std::min((q.nrec + 3) / 4, 256), 128, 0, st>>>(q);
  return cudaGetLastError();
}

cudaError_t f64_launch_step(int p, const F64Params &q, int nsm, cudaStream_t st) { SE2_DISPATCH(step, q, nsm, st) }
cudaError_t f64_launch_last(int p, const F64Params &q, double2 *v, double2 *a, cudaStream_t st) { SE2_DISPATCH(last, q, v, a, st) }
cudaError_t f64_launch_force(int p, const F64Params &q, double2 *f, cudaStream_t st) { SE2_DISPATCH(force, q, f, st) }
cudaError_t f64_launch_record(int p, const F64Params &q, cudaStream_t st) { SE2_DISPATCH(record, q, st) }

cudaError_t f64_launch_reciprocal(const double *mass, double *r, size_t n, int nsm, cudaStream_t st)
{
  f64_reciprocal<<<8 * nsm, 256, 0, st>>>(mass, r, n);
  return cudaGetLastError();
}

}  // namespace se2
