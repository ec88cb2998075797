// se2gpu_f32df.cu -- the two-float step kernels (every value of a step carried as a float pair,
// about 48 significant bits), degrees 1..8.  A translation unit of its own: the kernels are
// large and compile in parallel with the others, and this unit's constant tables (high and
// low parts of D and the GLL weights) are set here.
#include "se2gpu_f32df.cuh"

namespace se2p {

cudaError_t df_set_tables(int p, const double *D, const double *w1d)
{
  float dh[81] = {0}, dl[81] = {0}, wh[9] = {0}, wl[9] = {0};
  const int n1 = p + 1;
  for (int i = 0; i < n1 * n1; i++) {
    dh[i] = (float)D[i];
    dl[i] = (float)(D[i] - (double)dh[i]);
  }
  for (int i = 0; i < n1; i++) {
    wh[i] = (float)w1d[i];
    wl[i] = (float)(w1d[i] - (double)wh[i]);
  }
  const size_t od = sizeof(dh) * (p - 1), ow = sizeof(wh) * (p - 1);
  cudaError_t e = cudaMemcpyToSymbol(c_D, dh, sizeof(dh), od);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_Dl, dl, sizeof(dl), od);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_w, wh, sizeof(wh), ow);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_wl, wl, sizeof(wl), ow);
  return e;
}

namespace {

template <int P, int TE, int NT>
DfShape df_entry()
{
  static_assert(NT >= DfGeo<P, TE>::NE * (P + 1), "one (element, line) item per thread");
  return DfShape{P, TE, NT, DfGeo<P, TE>::SMEM, (const void *)df_step<P, TE, NT>, false};
}

// with a halo: registers sized for 2 CTAs per SM at most (1 with 384 threads or more): the pairs
// double most live values
template <int P, int TE, int NT>
DfShape halo_entry()
{
  typedef Layout<P, TE, true, 1, true> L;
  constexpr int MS = min_blocks(L::TOTAL);
  constexpr int M = (NT >= 384) ? 1 : (MS < 2 ? MS : 2);
  return DfShape{P, TE, NT, L::TOTAL, (const void *)persist_step<P, TE, NT, true, 1, M, true, false>, true};
}

const void *last_fn(int p)
{
  static const void *t[8] = {(const void *)df_last<1>, (const void *)df_last<2>, (const void *)df_last<3>,
                             (const void *)df_last<4>, (const void *)df_last<5>, (const void *)df_last<6>,
                             (const void *)df_last<7>, (const void *)df_last<8>};
  return t[p - 1];
}

template <int P>
cudaError_t record_t(const Params &prm, cudaStream_t st)
{
  persist_record<P, true><<<1, 128, 0, st>>>(prm);
  return cudaGetLastError();
}

}  // namespace

bool df_shape(int p, int config, DfShape *s)
{
#define SE2P_DF_ENTRY(P, TE, NT) df_entry<P, TE, NT>(),
#define SE2P_HALO_ENTRY(P, TE, NT) halo_entry<P, TE, NT>(),
  static const DfShape t[] = {SE2P_DF_CONFIGS(SE2P_DF_ENTRY, SE2P_HALO_ENTRY)};
#undef SE2P_HALO_ENTRY
#undef SE2P_DF_ENTRY
  int k = 0;
  for (const DfShape &e : t)
    if (e.p == p && k++ == config) {
      *s = e;
      return true;
    }
  return false;
}

cudaError_t df_launch(int p, int config, const EfParams &q, bool dependent, cudaStream_t st)
{
  DfShape s;
  if (!df_shape(p, config, &s) || s.halo) return cudaErrorInvalidValue;
  EfParams a = q;
  const int te = s.te * p, nbx = (q.p.nx_g + DF_LX - 1) / DF_LX, nblocks = nbx * ((q.p.ny_g + DF_LY - 1) / DF_LY);
  const bool last = q.mode == EF_LAST;
  void *step_args[] = {&a}, *last_args[] = {&a, (void *)&te, (void *)&nbx, (void *)&nblocks};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((last ? nblocks : q.p.ntiles) + (q.p.record ? 1 : 0));
  cfg.blockDim = dim3(last ? DF_LX * DF_LY : s.nt);
  cfg.dynamicSmemBytes = last ? 0 : s.smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = dependent ? 1 : 0;
  return last ? cudaLaunchKernelExC(&cfg, last_fn(p), last_args) : cudaLaunchKernelExC(&cfg, s.fn, step_args);
}

cudaError_t df_launch_record(int p, const Params &prm, cudaStream_t st)
{
  switch (p) {
    case 1: return record_t<1>(prm, st); case 2: return record_t<2>(prm, st);
    case 3: return record_t<3>(prm, st); case 4: return record_t<4>(prm, st);
    case 5: return record_t<5>(prm, st); case 6: return record_t<6>(prm, st);
    case 7: return record_t<7>(prm, st); case 8: return record_t<8>(prm, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace se2p
