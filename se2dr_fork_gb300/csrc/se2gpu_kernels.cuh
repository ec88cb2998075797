// se2gpu_kernels.cuh -- the FP32 internal force (AssembleLinearForm_ElastoDynamics2d,
// se2wave.c:1285-1429, in plain single precision) and the FP64 field norms, for sm_103a.
// Time stepping runs the kernels of se2gpu_f64.cuh and se2gpu_persist.cuh.
//
// Internal force.  A CTA owns a rectangle of GLL nodes: the nodes of a tile of TE x TE
// elements, minus the node line shared with the next tile.  The nodes on its left/bottom
// boundary line also receive forces from the element column/row of the neighbouring
// tile, so the CTA additionally evaluates that one-element halo.  Every owned node then
// sums the contributions of the 1, 2 or 4 elements touching it in ascending element
// order -- the order of the reference's VecSetValues(ADD) loop (1417) -- so there are no
// atomics and results are deterministic.  Phases (all in shared memory): load u of the
// node region; strain -> Hooke stress at every GLL point of every element of tile +
// halo (tensor-product gradient); weak divergence at the owned nodes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace se2 {

struct ForceParams {
  int mx, my, nx_g, ny_g;     // elements, nodes per row/column
  int ntx, nty;               // tile grid
  const float2 *u_in;
  float2 *f_out;
  const float *lam, *mu;      // per cell
  const float *J00, *J11, *iJ00, *iJ11;
  const float *D, *wq;        // (P+1)^2 tables
};

// tile geometry (elements per tile edge) per degree
template <int P> struct Tile { static constexpr int TE = (P == 1) ? 32 : (P == 2) ? 16 : (P == 3) ? 11 : (P == 4) ? 8
                                                       : (P == 5) ? 6 : (P == 6) ? 5 : 4; };

// shared-memory carve, identical on host and device
struct Smem {
  size_t U, S, W, D, total;
};
__host__ __device__ inline size_t se2_align16(size_t x) { return (x + 15) & ~size_t(15); }
template <int P>
__host__ __device__ inline Smem smem_layout()
{
  constexpr int TE = Tile<P>::TE, N1 = P + 1, NPE = N1 * N1;
  constexpr int RW = (TE + 1) * P + 1;
  constexpr int NE = (TE + 1) * (TE + 1);
  Smem s;
  size_t o = 0;
  s.U = o;  o = se2_align16(o + sizeof(float) * 2 * RW * RW);
  s.S = o;  o = se2_align16(o + sizeof(float) * 3 * NE * NPE);
  s.W = o;  o = se2_align16(o + sizeof(float) * NPE);
  s.D = o;  o = se2_align16(o + sizeof(float) * NPE);
  s.total = o;
  return s;
}

template <int P>
__global__ void __launch_bounds__(256)
force_kernel(const ForceParams prm)
{
  constexpr int TE = Tile<P>::TE, N1 = P + 1, NPE = N1 * N1;
  constexpr int NEMAX = (TE + 1) * (TE + 1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Smem L = smem_layout<P>();
  float2 *sU = reinterpret_cast<float2 *>(smem_raw + L.U);
  float *sSxx = reinterpret_cast<float *>(smem_raw + L.S);
  float *sSyy = sSxx + NEMAX * NPE;
  float *sSxy = sSyy + NEMAX * NPE;
  float *sW = reinterpret_cast<float *>(smem_raw + L.W);
  float *sD = reinterpret_cast<float *>(smem_raw + L.D);

  const int mx = prm.mx, my = prm.my, nx_g = prm.nx_g;
  const int tx = blockIdx.x % prm.ntx, ty = blockIdx.x / prm.ntx;
  const int ex0 = tx * TE, ex1 = min(ex0 + TE, mx);
  const int ey0 = ty * TE, ey1 = min(ey0 + TE, my);
  const int EX0 = max(ex0 - 1, 0), EY0 = max(ey0 - 1, 0);
  const int NEX = ex1 - EX0, NEY = ey1 - EY0;
  const int RX0 = EX0 * P, RY0 = EY0 * P;
  const int RW = NEX * P + 1, RH = NEY * P + 1;
  const int X0 = ex0 * P, Y0 = ey0 * P;
  const int OW = (ex1 - ex0) * P + (ex1 == mx ? 1 : 0);
  const int OH = (ey1 - ey0) * P + (ey1 == my ? 1 : 0);

  // ---- phase 1: load -------------------------------------------------
  for (int idx = threadIdx.x; idx < RW * RH; idx += blockDim.x) {
    const int ry = idx / RW, rx = idx - ry * RW;
    sU[idx] = prm.u_in[(size_t)(RY0 + ry) * nx_g + RX0 + rx];
  }
  for (int i = threadIdx.x; i < NPE; i += blockDim.x) { sW[i] = prm.wq[i]; sD[i] = prm.D[i]; }
  __syncthreads();

  // ---- phase 2: stress at every GLL point of tile + halo -------------
  const int NEL = NEX * NEY;
  for (int idx = threadIdx.x; idx < NEL * NPE; idx += blockDim.x) {
    const int el = idx / NPE, q = idx - el * NPE;
    const int ecy = el / NEX, ecx = el - ecy * NEX;
    const int qj = q / N1, qi = q - qj * N1;
    const int ex = EX0 + ecx, ey = EY0 + ecy;
    const float2 *ue = sU + (ecy * P) * RW + ecx * P;   // local node (0,0)
    const size_t cell = (size_t)ey * mx + ex;
    const float lam = prm.lam[cell], mu = prm.mu[cell];
    float gx_ux = 0.f, gx_uy = 0.f, gy_ux = 0.f, gy_uy = 0.f;
#pragma unroll
    for (int k = 0; k < N1; k++) {
      const float dxk = sD[qi * N1 + k], dyk = sD[qj * N1 + k];
      const float2 ur = ue[qj * RW + k];   // row through q
      const float2 uc = ue[k * RW + qi];   // column through q
      gx_ux = fmaf(dxk, ur.x, gx_ux);
      gx_uy = fmaf(dxk, ur.y, gx_uy);
      gy_ux = fmaf(dyk, uc.x, gy_ux);
      gy_uy = fmaf(dyk, uc.y, gy_uy);
    }
    const float ix = prm.iJ00[ex], iy = prm.iJ11[ey];
    const float e0 = ix * gx_ux, e1 = iy * gy_uy, e2 = fmaf(ix, gx_uy, iy * gy_ux);
    const float c11 = fmaf(2.f, mu, lam);
    const float nfac = -(prm.J00[ex] * prm.J11[ey]) * sW[q];
    sSxx[idx] = nfac * fmaf(c11, e0, lam * e1);
    sSyy[idx] = nfac * fmaf(lam, e0, c11 * e1);
    sSxy[idx] = nfac * (mu * e2);
  }
  __syncthreads();

  // ---- phase 3: divergence, ordered element sum -----------------------
  for (int o = threadIdx.x; o < OW * OH; o += blockDim.x) {
    const int oy = o / OW, ox = o - oy * OW;
    const int X = X0 + ox, Y = Y0 + oy;
    float fx = 0.f, fy = 0.f;
    const int eyA = (Y % P == 0) ? Y / P - 1 : Y / P, exA = (X % P == 0) ? X / P - 1 : X / P;
    const int eyB = Y / P, exB = X / P;
    for (int ey = eyA; ey <= eyB; ey++) {
      if (ey < 0 || ey >= my) continue;
      for (int ex = exA; ex <= exB; ex++) {
        if (ex < 0 || ex >= mx) continue;
        const int el = (ey - EY0) * NEX + ex - EX0;
        const int a = X - ex * P, b = Y - ey * P;
        const float *Sxx = sSxx + el * NPE, *Syy = sSyy + el * NPE, *Sxy = sSxy + el * NPE;
        float rx = 0.f, ry = 0.f, cx = 0.f, cy = 0.f;
#pragma unroll
        for (int k = 0; k < N1; k++) {
          const float dxa = sD[k * N1 + a], dyb = sD[k * N1 + b];
          rx = fmaf(dxa, Sxx[k + b * N1], rx);
          ry = fmaf(dxa, Sxy[k + b * N1], ry);
          cx = fmaf(dyb, Sxy[a + k * N1], cx);
          cy = fmaf(dyb, Syy[a + k * N1], cy);
        }
        const float ix = prm.iJ00[ex], iy = prm.iJ11[ey];
        fx += fmaf(ix, rx, iy * cx);
        fy += fmaf(ix, ry, iy * cy);
      }
    }
    prm.f_out[(size_t)Y * nx_g + X] = make_float2(fx, fy);
  }
}

// ---- norms: per-block partials, then a single-block fixed-order finish ----
static __global__ void norms_partial(const double *u, const double *v, long n, double *part)
{
  __shared__ double s[6][256];
  double umax = -1.0e308, umin = 1.0e308, uss = 0.0, vmax = -1.0e308, vmin = 1.0e308, vss = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double a = u[i], b = v[i];
    umax = fmax(umax, a); umin = fmin(umin, a); uss += a * a;
    vmax = fmax(vmax, b); vmin = fmin(vmin, b); vss += b * b;
  }
  s[0][threadIdx.x] = umax; s[1][threadIdx.x] = umin; s[2][threadIdx.x] = uss;
  s[3][threadIdx.x] = vmax; s[4][threadIdx.x] = vmin; s[5][threadIdx.x] = vss;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      const int t = threadIdx.x;
      s[0][t] = fmax(s[0][t], s[0][t + w]); s[1][t] = fmin(s[1][t], s[1][t + w]); s[2][t] += s[2][t + w];
      s[3][t] = fmax(s[3][t], s[3][t + w]); s[4][t] = fmin(s[4][t], s[4][t + w]); s[5][t] += s[5][t + w];
    }
    __syncthreads();
  }
  if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = s[threadIdx.x][0];
}

}  // namespace se2
