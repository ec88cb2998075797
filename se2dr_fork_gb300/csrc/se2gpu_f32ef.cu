// se2gpu_f32ef.cu -- plain and Kahan step kernels without a halo, degrees 1..8 (a translation unit with
// its own constant tables, compiled in parallel with the others).
#include "se2gpu_f32ef.cuh"

namespace se2p {

cudaError_t ef_set_tables(int p, const double *D, const double *w1d)
{
  float d[81] = {0}, w[9] = {0};
  const int n1 = p + 1;
  for (int i = 0; i < n1 * n1; i++) d[i] = (float)D[i];
  for (int i = 0; i < n1; i++) w[i] = (float)w1d[i];
  const cudaError_t e = cudaMemcpyToSymbol(c_D, d, sizeof(d), sizeof(d) * (p - 1));
  return e != cudaSuccess ? e : cudaMemcpyToSymbol(c_w, w, sizeof(w), sizeof(w) * (p - 1));
}

namespace {
template <int P, int TE, int NT>
EfShape entry()
{
  static_assert(NT >= TE * TE * (P + 1), "one (element, line) item per thread");
  return EfShape{P, TE, NT, {ef_smem(P, TE, false, Xch<P, false>::XS), ef_smem(P, TE, true, Xch<P, true>::XS)},
                 {(const void *)ef_step<P, TE, NT, false>, (const void *)ef_step<P, TE, NT, true>}};
}
}  // namespace

bool ef_shape(int p, int k, EfShape *s)
{
#define SE2P_EF_ENTRY(P, TE, NT) entry<P, TE, NT>(),
  static const EfShape t[] = {SE2P_EF_CONFIGS(SE2P_EF_ENTRY)};
#undef SE2P_EF_ENTRY
  for (const EfShape &e : t)
    if (e.p == p && k-- == 0) {
      *s = e;
      return true;
    }
  return false;
}

cudaError_t ef_launch(int p, int k, bool kahan, const EfParams &q, bool dependent, cudaStream_t st)
{
  EfShape s;
  if (!ef_shape(p, k, &s)) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(q.p.ntiles + (q.p.record ? 1 : 0));
  cfg.blockDim = dim3(s.nt);
  cfg.dynamicSmemBytes = s.smem[kahan ? 1 : 0];
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = dependent ? 1 : 0;
  EfParams a = q;
  void *args[] = {&a};
  return cudaLaunchKernelExC(&cfg, s.fn[kahan ? 1 : 0], args);
}

}  // namespace se2p
