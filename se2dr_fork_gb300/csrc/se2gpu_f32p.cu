// se2gpu_f32p.cu -- persistent TMA-pipelined FP32 kernels (plain / Kahan; the two-float mode is
// in se2gpu_f32df.cu), degrees 1..8, the tile configurations the autotuner chooses from, and
// their host-side helpers (tensor maps, constant tables, norms of the leapfrog state).
#include <cudaTypedefs.h>

#include <algorithm>

#include "se2gpu_f32df_launch.h"
#include "se2gpu_f32ef_launch.h"
#include "se2gpu_persist.cuh"
#include "se2gpu_persist_launch.h"

namespace se2p {

cudaError_t set_tables(int p, const double *D, const double *w1d)
{
  float d[81] = {0}, w[9] = {0};
  const int n1 = p + 1;
  for (int i = 0; i < n1 * n1; i++) d[i] = (float)D[i];
  for (int i = 0; i < n1; i++) w[i] = (float)w1d[i];
  cudaError_t e = cudaMemcpyToSymbol(c_D, d, sizeof(d), sizeof(d) * (p - 1));
  if (e != cudaSuccess) return e;
  e = cudaMemcpyToSymbol(c_w, w, sizeof(w), sizeof(w) * (p - 1));
  if (e != cudaSuccess) return e;
  e = df_set_tables(p, D, w1d);
  return e != cudaSuccess ? e : ef_set_tables(p, D, w1d);
}

// ---- one configuration = (degree, elements per tile edge, threads) ----------
struct Entry {
  int p, te, nt, nob;
  size_t smem[2];                 // [kahan]
  size_t bsmem[2];                // batched kernel [kahan]
  const void *fn[2];              // persist_step<...> [kahan]
  const void *bfn[2];             // persist_batch<...> [kahan]
};

template <int P, int TE, int NT, int NOB = owned_buffers(P), int MINB = 0, bool WE = false, int NST = 2>
static Entry entry()
{
  constexpr int M0 = MINB ? MINB : min_blocks(Layout<P, TE, false, NOB, false, true>::TOTAL);
  constexpr int M1 = MINB ? MINB : min_blocks(Layout<P, TE, true, NOB, false, true>::TOTAL);
  constexpr int B0 = MINB ? MINB : min_blocks(Layout<P, TE, false, NOB>::BATCH_TOTAL);
  constexpr int B1 = MINB ? MINB : min_blocks(Layout<P, TE, true, NOB>::BATCH_TOTAL);
  Entry e;
  e.p = P; e.te = TE; e.nt = NT; e.nob = NOB;
  e.smem[0] = NST == 2 ? Layout<P, TE, false, NOB, false, true>::TOTAL : Layout<P, TE, false, NOB, false, true>::TOTAL1;
  e.smem[1] = NST == 2 ? Layout<P, TE, true, NOB, false, true>::TOTAL : Layout<P, TE, true, NOB, false, true>::TOTAL1;
  e.bsmem[0] = Layout<P, TE, false, NOB>::BATCH_TOTAL;
  e.bsmem[1] = Layout<P, TE, true, NOB>::BATCH_TOTAL;
  e.fn[0] = (const void *)persist_step<P, TE, NT, false, NOB, M0, false, WE, NST>;
  e.fn[1] = (const void *)persist_step<P, TE, NT, true, NOB, M1, false, WE, NST>;
  e.bfn[0] = (const void *)persist_batch<P, TE, NT, false, NOB, B0, WE>;
  e.bfn[1] = (const void *)persist_batch<P, TE, NT, true, NOB, B1, WE>;
  return e;
}

static const Entry *table(int *n)
{
#define SE2P_ENTRY(P, TE, NT, NOB, MINB, WE) entry<P, TE, NT, (NOB) ? (NOB) : owned_buffers(P), MINB, (WE) == 1, (WE) == 2 ? 1 : 2>(),
  static Entry t[] = {SE2P_CONFIGS(SE2P_ENTRY)};
#undef SE2P_ENTRY
  *n = (int)(sizeof(t) / sizeof(t[0]));
  return t;
}

static const Entry *find(int p, int config)
{
  int n, k = 0;
  const Entry *t = table(&n);
  for (int i = 0; i < n; i++)
    if (t[i].p == p) {
      if (k == config) return &t[i];
      k++;
    }
  return nullptr;
}

// the tiles for meshes of many tiles.  Plain and Kahan: per degree the one the autotuner
// measured fastest on GB300 at about 16M nodes (and, at degree 4, at the 2048^2 workload; the
// plain mode at degree 8 runs 4 x 4 tiles: 83 against 93 us a step at 5M nodes, 7.0 against 9.6 at
// 260000), and smaller tiles on meshes that these divide into about one per SM (us a step: degree 6,
// 47 x 47 elements 6.43 -> 5.91; plain degree 8, 31 x 31 6.52 -> 5.60).  On still smaller ones
// first_config goes over to the step without a halo (se2gpu_f32ef.cuh; Kahan, 80000 nodes, halo / not:
// degree 1 5.2 / 6.9, 2 5.3 / 5.4, 3 5.2 / 5.2, 4 5.8 / 5.5, 5 5.9 / 6.3, 6 5.9 / 6.1, 7 7.2 / 5.9, 8
// 6.5 / 7.6).  Two-float: small tiles with a thread per node while a few of them fill an SM, then
// those with the fewest idle threads, then (degrees 2 and 3) the halo kernel; the lines lie where
// the times cross (us a step at 20000 / 80000 / 260000 / 1M nodes): degree 2 6 x 6 5.1 / 8.7 / 20.6 / 81,
// 8 x 8 6.8 / 10.1 / 20.2 / 78, halo 8.6 / 9.1 / 25.4 / 75; 3 4 x 4 with 192 threads 5.6 / 8.1 / 20.5 / 78,
// with 64 7.7 / 9.0 / 19.5 / 72, halo 7.7 / 9.9 / 22.0 / 69; 4 3 x 3 7.8 / 9.2 / 25 / 96, 5 x 5 10.6 / 11.1 /
// 20 / 70; 5 2 x 2 8.6 / 10.8 / 24.6 / 95, 4 x 4 12.7 / 12.8 / 22.1 / 74; 6 2 x 2 10.2 / 18.1 / 51 / 196, 3 x 3
// 14.2 / 13.4 / 21.4 / 82, 6 x 6 19.1 / 17.9 / 24.9 / 79; 7 2 x 2 11.9 / 20.2 / 48 / 177, 4 x 4 18.4 / 17.5 /
// 24.9 / 81; 8 1 x 1 12.4 / 23.5 / 69 / 247, 3 x 3 17.5 / 17.0 / 29 / 100, 5 x 5 24 / 24 / 34 / 92.
// mx = 0: the large-mesh choice (the ensemble's, whose shots share one).
int default_config(int p, int mode, int mx, int my, int nsm)
{
  if (p < 1 || p > 8) return 0;
  auto tiles = [&](int config) {
    const Entry *e = find(p, config);
    DfShape df;
    const int te = (mode == MODE_DF && df_shape(p, config, &df)) ? df.te : e ? e->te : 0;
    return (mx == 0 || !te) ? 1L << 40 : (long)((mx + te - 1) / te) * ((my + te - 1) / te);
  };
  if (mode == MODE_DF) {
    switch (p) {
      case 1: return tiles(1) <= nsm ? 1 : 0;
      case 2: return tiles(2) <= 4L * nsm ? 2 : tiles(1) <= 16L * nsm ? 1 : 0;
      case 3: return tiles(2) <= 4L * nsm ? 2 : tiles(1) <= 28L * nsm ? 1 : 0;
      case 4: return tiles(4) <= 4L * nsm ? 4 : 0;
      case 5: return tiles(2) <= 6L * nsm ? 2 : 0;
      case 6: return tiles(2) <= 2L * nsm ? 2 : tiles(0) < 4L * nsm ? 1 : 0;
      case 7: return tiles(2) <= 2L * nsm ? 2 : 0;
      default: return tiles(2) <= 5L * nsm ? 2 : tiles(0) < 2L * nsm ? 1 : 0;
    }
  }
  static const int best[8] = {2, 0, 2, 1, 2, 0, 2, 1}, small[8] = {1, 2, 2, 1, 1, 1, 2, 1};
  if (tiles(small[p - 1]) <= ((p == 2 || p == 8) ? 2 : 1) * (long)nsm) return small[p - 1];
  return (p == 8 && mode == MODE_PLAIN) ? 0 : best[p - 1];
}

int num_configs(int p)
{
  int n, k = 0;
  const Entry *t = table(&n);
  for (int i = 0; i < n; i++) k += (t[i].p == p);
  return k;
}

int auto_config(int p, int mode) { return default_config(p, mode, 0, 0, 1); }

// The tiles of a new handle (and of the number auto_config): the step without a halo on a small mesh, up
// to few[] of its tiles per SM, and at two degrees other tiles than default_config's where the rounds
// that the resident CTAs need, times the elements of a tile with its halo, say that these take less.
// us a step, Kahan / plain.  Degree 4: 6 x 6 while one per SM holds the mesh (71 x 71 elements 6.0 ->
// 5.3 / 5.5 -> 5.0); 8 x 8 with one region stage, two CTAs per SM, in up to two rounds (128 x 128 8.7 -> 7.5
// / 8.0 -> 6.6; 177 x 177 13.0 -> 12.2 / 11.5 -> 10.6; but 500 x 500 68 / 76: nothing is copied ahead).
// Degree 7: 5 x 5 with one region stage, which leaves two (plain: three) CTAs per SM instead of one
// (85 x 85 10.7 -> 9.1 / 10.7 -> 8.1; 143 x 143 22.5 -> 19.5 / 18.3 -> 15.9; 571 x 571 267 -> 254 / 207 -> 184; with both stages
// 5 x 5 takes 284 / 200 there).
// The tiles of the other degrees' large meshes leave two or three CTAs per SM with both stages; none with one was
// built for them.
int first_config(int p, int mode, int mx, int my, int nsm)
{
  static const int few[8] = {3, 2, 2, 4, 3, 2, 3, 3};
  if (mode == MODE_DF || mx == 0) return default_config(p, mode, mx, my, nsm);
  auto tiles = [&](int te) { return (long)((mx + te - 1) / te) * ((my + te - 1) / te); };
  auto cost = [&](int te, int per_sm) {
    const long slots = (long)per_sm * nsm;
    return (tiles(te) + slots - 1) / slots * (te + 1) * (te + 1);
  };
  EfShape ef;
  if (ef_shape(p, 0, &ef) && tiles(ef.te) <= few[p - 1] * (long)nsm) return num_configs(p);
  if (p == 4 && tiles(6) <= nsm) return 2;
  if (p == 4 && tiles(8) <= 4L * nsm && cost(8, 2) < cost(7, 2)) return 6;
  const int per_sm = (mode == MODE_KAHAN) ? 2 : 3;
  if (p == 7 && 10 * cost(5, per_sm) <= 11 * cost(4, per_sm)) return 3;   // (5 x 5 has the smaller halo)
  return default_config(p, mode, mx, my, nsm);
}

int num_configs(int p, int mode)
{
  EfShape e;
  DfShape d;
  int n = 0;
  if (mode == MODE_DF) {
    while (df_shape(p, n, &d)) n++;
    return n;
  }
  while (ef_shape(p, n, &e)) n++;
  return num_configs(p) + n;
}

// a configuration without a halo, of any mode
static bool no_halo(int p, int config, int mode, DfShape *s)
{
  if (mode == MODE_DF) return df_shape(p, config, s) && !s->halo;
  EfShape e;
  if (config < num_configs(p) || !ef_shape(p, config - num_configs(p), &e)) return false;
  const int k = mode ? 1 : 0;
  *s = DfShape{p, e.te, e.nt, e.smem[k], e.fn[k], false};
  return true;
}

cudaError_t launch_no_halo(int p, int config, int mode, const EfParams &q, bool dependent, cudaStream_t st)
{
  if (mode == MODE_DF) return df_launch(p, config, q, dependent, st);
  return ef_launch(p, config - num_configs(p), mode == MODE_KAHAN, q, dependent, st);
}

int config_shape(int p, int config, int mode, TileShape *s)
{
  const Entry *e = find(p, config);
  DfShape df;
  if (no_halo(p, config, mode, &df)) {
    *s = TileShape{};   // (no tensor maps; the state of the tile is held once)
    s->owned_buffers = 1;
    s->tex = s->tey = df.te;
    s->nt = df.nt;
    s->smem = df.smem;
    return 0;
  }
  if (!e || (mode == MODE_DF && !df_shape(p, config, &df))) return -1;
  const int te = (mode == MODE_DF) ? df.te : e->te;
  s->halo = true;
  s->tex = s->tey = te;
  s->nt = (mode == MODE_DF) ? df.nt : e->nt;
  s->region_w = round_up((te + 1) * p + 2 + ((p & 1) ? 2 : 0), 2);
  s->region_h = (te + 1) * p + 1;
  s->own_w = round_up(te * p + 2, 2);
  s->own_h = te * p + 1;
  s->cell_box = te + 1;
  s->minv_w = round_up(te * p + 1 + 4, 4);
  s->owned_buffers = (mode == MODE_DF) ? 1 : e->nob;
  s->smem = (mode == MODE_DF) ? df.smem : e->smem[mode ? 1 : 0];
  return 0;
}

static cudaError_t prepare_kernel(const void *fn, size_t smem)
{
  const cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return r != cudaSuccess ? r : cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}

cudaError_t prepare(int p, int config, int mode)
{
  const Entry *e = find(p, config);
  const int k = mode ? 1 : 0;
  DfShape s = {};
  if (no_halo(p, config, mode, &s) || (mode == MODE_DF && df_shape(p, config, &s))) return prepare_kernel(s.fn, s.smem);
  if (!e || mode == MODE_DF) return cudaErrorInvalidValue;
  const cudaError_t r = prepare_kernel(e->fn[k], e->smem[k]);
  return r != cudaSuccess ? r : prepare_kernel(e->bfn[k], e->bsmem[k]);
}

int occupancy(int p, int config, int mode, bool batch)
{
  const Entry *e = find(p, config);
  int n = 0;
  const int k = mode ? 1 : 0;
  DfShape s = {};
  if (e) s = DfShape{p, e->te, e->nt, (batch ? e->bsmem : e->smem)[k], (batch ? e->bfn : e->fn)[k], true};
  if (!batch && mode == MODE_DF) df_shape(p, config, &s);
  if (!batch) no_halo(p, config, mode, &s);
  if (!s.fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, s.fn, s.nt, s.smem) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return std::min(n, 3);   // the persistent grid's CTAs per SM: what the tile configurations are sized for
}

// a launch that may begin (its set-up before cudaGridDependencySynchronize) while the launch
// before it on the stream drains: about 2 us of every short step
static cudaError_t launch(const void *fn, int grid, int threads, void **args, size_t smem, bool dependent, cudaStream_t st)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

cudaError_t launch_step(int p, int config, int mode, const CUtensorMap *maps, const Params &prm, int grid,
                        bool dependent, cudaStream_t st)
{
  const Entry *e = find(p, config);
  if (!e) return cudaErrorInvalidValue;
  DfShape s{p, e->te, e->nt, e->smem[mode ? 1 : 0], e->fn[mode ? 1 : 0], true};
  if (mode == MODE_DF && (!df_shape(p, config, &s) || !s.halo)) return cudaErrorInvalidValue;   // (df_launch)
  Params pc = prm;
  CUtensorMap m0 = maps[0], m1 = maps[1], m2 = maps[2], m3 = maps[3], m4 = maps[4], m5 = maps[5];
  void *args[] = {&m0, &m1, &m2, &m3, &m4, &m5, &pc};
  return launch(s.fn, grid, s.nt, args, s.smem, dependent, st);
}

cudaError_t launch_batch(int p, int config, bool kahan, const BatchArgs &ba, int grid, bool dependent, cudaStream_t st)
{
  const Entry *e = find(p, config);
  if (!e) return cudaErrorInvalidValue;
  BatchArgs a = ba;
  void *args[] = {&a};
  return launch(e->bfn[kahan ? 1 : 0], grid, e->nt, args, e->bsmem[kahan ? 1 : 0], dependent, st);
}

template <int P>
static cudaError_t record_batch_t(const Params *shots, int nshots, int kblk, cudaStream_t st)
{
  persist_record_batch<P><<<nshots, 128, 0, st>>>(shots, nshots, kblk);
  return cudaGetLastError();
}
cudaError_t launch_record_batch(int p, const Params *shots, int nshots, int kblk, cudaStream_t st)
{
  if (nshots <= 0) return cudaSuccess;
  switch (p) {
    case 1: return record_batch_t<1>(shots, nshots, kblk, st); case 2: return record_batch_t<2>(shots, nshots, kblk, st);
    case 3: return record_batch_t<3>(shots, nshots, kblk, st); case 4: return record_batch_t<4>(shots, nshots, kblk, st);
    case 5: return record_batch_t<5>(shots, nshots, kblk, st); case 6: return record_batch_t<6>(shots, nshots, kblk, st);
    case 7: return record_batch_t<7>(shots, nshots, kblk, st); case 8: return record_batch_t<8>(shots, nshots, kblk, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int P>
static cudaError_t record_t(const Params &prm, cudaStream_t st)
{
  persist_record<P><<<1, 128, 0, st>>>(prm);
  return cudaGetLastError();
}
cudaError_t launch_record(int p, const Params &prm, cudaStream_t st, bool df)
{
  if (df) return df_launch_record(p, prm, st);
  switch (p) {
    case 1: return record_t<1>(prm, st); case 2: return record_t<2>(prm, st);
    case 3: return record_t<3>(prm, st); case 4: return record_t<4>(prm, st);
    case 5: return record_t<5>(prm, st); case 6: return record_t<6>(prm, st);
    case 7: return record_t<7>(prm, st); case 8: return record_t<8>(prm, st);
    default: return cudaErrorInvalidValue;
  }
}

// tensor map of one padded float2 field, box (bw, bh) nodes
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

static int encoder()
{
  if (!g_encode) {
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return -1;
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  return 0;
}

int make_map(CUtensorMap *map, void *base, int nx, int ny, int pitch, int bw, int bh)
{
  if (encoder()) return -1;
  cuuint64_t dims[2] = {(cuuint64_t)nx, (cuuint64_t)ny};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * 8};
  cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(int)r - 1000;
}

int make_map_f32(CUtensorMap *map, void *base, int nx, int ny, int pitch, int bw, int bh)
{
  if (encoder()) return -1;
  cuuint64_t dims[2] = {(cuuint64_t)nx, (cuuint64_t)ny};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * 4};
  cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(int)r - 1000;
}

int make_map_cells(CUtensorMap *map, void *base, int mx, int my, int box)
{
  if (encoder()) return -1;
  cuuint64_t dims[3] = {4, (cuuint64_t)mx, (cuuint64_t)my};
  cuuint64_t strides[2] = {16, (cuuint64_t)mx * 16};
  cuuint32_t bx[3] = {4, (cuuint32_t)box, (cuuint32_t)box};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, bx, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(int)r - 1000;
}

// norms of (u_k, v_k) recovered from the leapfrog state in FP64:
// u_k = (u - cu) - dt (w - cw),  v_k = (w - cw) - dt/2 a_k
__global__ void norms_leapfrog(const float2 *u, const float2 *w, const float2 *cu, const float2 *cw, const float2 *a,
                               const float2 *al, int nx, int ny, int pitch, double dt, double half_dt, double *part)
{
  __shared__ double s[6][256];
  double umax = -1.0e308, umin = 1.0e308, uss = 0.0, vmax = -1.0e308, vmin = 1.0e308, vss = 0.0;
  const long n = (long)nx * ny;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const long y = i / nx, x = i - y * nx, k = y * pitch + x;
    const float2 uu = u[k], ww = w[k], aa = a[k], aal = al ? al[k] : make_float2(0.f, 0.f);
    const float2 cuu = cu ? cu[k] : make_float2(0.f, 0.f), cww = cw ? cw[k] : make_float2(0.f, 0.f);
    const double wx = (double)ww.x - (double)cww.x, wy = (double)ww.y - (double)cww.y;
    const double ux = ((double)uu.x - (double)cuu.x) - dt * wx, uy = ((double)uu.y - (double)cuu.y) - dt * wy;
    const double vx = wx - half_dt * ((double)aa.x + (double)aal.x), vy = wy - half_dt * ((double)aa.y + (double)aal.y);
    umax = fmax(umax, fmax(ux, uy)); umin = fmin(umin, fmin(ux, uy)); uss += ux * ux + uy * uy;
    vmax = fmax(vmax, fmax(vx, vy)); vmin = fmin(vmin, fmin(vx, vy)); vss += vx * vx + vy * vy;
  }
  s[0][threadIdx.x] = umax; s[1][threadIdx.x] = umin; s[2][threadIdx.x] = uss;
  s[3][threadIdx.x] = vmax; s[4][threadIdx.x] = vmin; s[5][threadIdx.x] = vss;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      const int t = threadIdx.x;
      s[0][t] = fmax(s[0][t], s[0][t + h]); s[1][t] = fmin(s[1][t], s[1][t + h]); s[2][t] += s[2][t + h];
      s[3][t] = fmax(s[3][t], s[3][t + h]); s[4][t] = fmin(s[4][t], s[4][t + h]); s[5][t] += s[5][t + h];
    }
    __syncthreads();
  }
  if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = s[threadIdx.x][0];
}

cudaError_t launch_norms(const float2 *u, const float2 *w, const float2 *cu, const float2 *cw, const float2 *a,
                         const float2 *al, int nx, int ny, int pitch, double dt, double *part, int nblocks,
                         cudaStream_t st)
{
  norms_leapfrog<<<nblocks, 256, 0, st>>>(u, w, cu, cw, a, al, nx, ny, pitch, dt, 0.5 * dt, part);
  return cudaGetLastError();
}

// The step kernels' bounded wait and error flag, on an mbarrier that nothing arrives
// at: the wait gives up after EXPIRY_TEST_POLLS polls and the kernel raises the flag,
// as a step kernel does when its tile copies never land.  No copy is in flight, so
// the CTA exits normally.  ns[0] = the wait's duration (globaltimer).
__global__ void wait_expiry_test(int *err, unsigned long long *ns)
{
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x != 0) return;
  const uint32_t b = smem_u32(&bar);
  mbar_init(b, 1);
  fence_barrier_init();
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  const bool ok = mbar_wait_bounded<EXPIRY_TEST_POLLS>(b, 0);
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  if (!ok) atomicExch(err, 1);
  ns[0] = t1 - t0;
}

cudaError_t launch_wait_expiry_test(int *err, unsigned long long *ns, cudaStream_t st)
{
  wait_expiry_test<<<1, 32, 0, st>>>(err, ns);
  return cudaGetLastError();
}

}  // namespace se2p
