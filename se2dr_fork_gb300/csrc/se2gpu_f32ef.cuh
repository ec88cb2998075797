// se2gpu_f32ef.cuh -- the plain and Kahan FP32 step without a halo of elements, for sm_103a.
//
// The arithmetic of se2gpu_persist.cuh's tile body, with the split of the two-float step
// (se2gpu_f32df.cuh): a launch finishes the previous step at the nodes of its tile, from the element
// forces in memory, then leaves the element forces of the new state there (8 (p+1)^2 bytes per
// element, two buffers).  A block of n steps is EF_START, n - 1 times EF_MIDDLE, EF_LAST.
//
// For small meshes, where the step is a chain of latencies: no TMA hop, no halo, so tiles down to one
// element spread over the SMs, and about a thread per node.  Kahan, us a step with 16 receivers,
// tile body -> this (2000 / 20000 nodes): degree 1 4.2 -> 3.6 / 4.2 -> 3.9, 2 5.6 -> 4.3 / 4.7 -> 4.1,
// 3 6.0 -> 4.6 / 4.9 -> 4.6, 4 8.4 -> 4.8 / 6.7 -> 4.7, 5 8.3 -> 5.0 / 6.4 -> 5.2, 6 8.6 -> 5.2 / 6.5 -> 5.2,
// 7 9.7 -> 5.5 / 7.8 -> 5.3, 8 9.3 -> 5.5 / 6.8 -> 5.9.  From about 100000 nodes on it loses (degree 4
// 8.4 / 8.9 at 260000 with its best tiles, 69 / 116 at 4M: there the forces' traffic counts).
#pragma once
#include "se2gpu_f32ef_launch.h"
#include "se2gpu_persist.cuh"

namespace se2p {

// what a node of the step to finish reads, loaded one node ahead of its use
template <bool KAHAN>
struct EfNode {
  float2 u, w, g[4];   // g: the forces of the elements around it, in ascending element order
  float minv;
  float2 cu[KAHAN], cw[KAHAN];
};
template <>
struct EfNode<false> {
  float2 u, w, g[4];
  float minv;
};

template <int P, int TE, int NT, bool KAHAN>
__global__ void __launch_bounds__(NT, ef_min_blocks(P, NT)) ef_step(const EfParams dp)
{
  constexpr int N1 = P + 1, NPE = N1 * N1, RW = TE * P + 1, NE = TE * TE;
  constexpr int XS = Xch<P, KAHAN>::XS, RS = Xch<P, KAHAN>::RS;
  const Params &prm = dp.p;
  const float *D = c_D[P - 1], *W = c_w[P - 1];
  extern __shared__ __align__(128) unsigned char smem[];
  float2 *X1 = reinterpret_cast<float2 *>(smem), *X2 = X1 + NE * XS, *sU = X2 + NE * XS, *sC = sU + RW * RW;
  cudaGridDependencySynchronize();
  if ((int)blockIdx.x >= prm.ntiles) {   // (one more CTA: the receivers of the step before)
    if (prm.record) sample_rows<P>(prm, prm.rbuf_in, prm.trace_row);
    return;
  }
  const int ty = blockIdx.x / prm.ntx, tx = blockIdx.x - ty * prm.ntx;
  const int ex0 = tx * TE, ey0 = ty * TE, nex = min(TE, prm.mx - ex0), ney = min(TE, prm.my - ey0);
  const int X0 = ex0 * P, Y0 = ey0 * P, pitch = prm.pitch;

  // ---- the tile's nodes: finish the previous step (a node line shared with the next tile belongs to
  // that one, which writes it)
  const int own_w = nex * P + (ex0 + nex == prm.mx ? 1 : 0), own_h = ney * P + (ey0 + ney == prm.my ? 1 : 0);
  const int4 bnd = prm.tile_bounds[blockIdx.x];
  const int s0 = bnd.x, s1 = bnd.y, r0 = bnd.z, r1 = bnd.w;
  const float dt = prm.dt, half_dt = prm.half_dt;
  auto load = [&](int i, EfNode<KAHAN> &d) {
    const int ry = i / RW, rx = i - ry * RW;
    if (i >= RW * RW || rx > nex * P || ry > ney * P) return;
    const int X = X0 + rx, Y = Y0 + ry;
    const size_t n = (size_t)Y * pitch + X;
    d.u = dp.u_in[n];
    if constexpr (KAHAN) d.cu[0] = dp.cu_in[n];
    if (dp.mode == EF_START) return;
    d.w = dp.w_in[n];
    if constexpr (KAHAN) d.cw[0] = dp.cw_in[n];
    d.minv = prm.minv[n];
    const NodePos<P> c(prm.mx, prm.my, X, Y);
    const float2 *ef = static_cast<const float2 *>(dp.ef_in) + ((ptrdiff_t)c.ey * prm.mx + c.ex) * NPE + c.ix + c.iy * N1;
    if (c.bot && c.lft) d.g[0] = ef[-(ptrdiff_t)(prm.mx + 1) * NPE + P + P * N1];
    if (c.bot && c.in_x) d.g[1] = ef[-(ptrdiff_t)prm.mx * NPE + P * N1];
    if (c.lft && c.in_y) d.g[2] = ef[-(ptrdiff_t)NPE + P];
    if (c.in_x && c.in_y) d.g[3] = ef[0];
  };
  EfNode<KAHAN> next;
  load(threadIdx.x, next);
#pragma unroll 1
  for (int i = threadIdx.x; i < RW * RW; i += NT) {
    const EfNode<KAHAN> d = next;
    load(i + NT, next);
    const int ry = i / RW, rx = i - ry * RW;
    const bool own = rx < own_w && ry < own_h;
    if (rx > nex * P || ry > ney * P || (dp.mode == EF_LAST && !own)) continue;
    const int X = X0 + rx, Y = Y0 + ry;
    const size_t n = (size_t)Y * pitch + X;
    float2 u = d.u, w = d.w, cu = make_float2(0.f, 0.f), cw = cu;
    if constexpr (KAHAN) {
      cu = d.cu[0];
      cw = d.cw[0];
    }
    if (dp.mode != EF_START) {
      float fx = 0.f, fy = 0.f;
      {
        const NodePos<P> c(prm.mx, prm.my, X, Y);
        const bool have[4] = {c.bot && c.lft, c.bot && c.in_x, c.lft && c.in_y, c.in_x && c.in_y};
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (have[k]) {
            fx += d.g[k].x;
            fy += d.g[k].y;
          }
      }
      SE2P_COLD for (int q = s0; q < s1; q++) {
        const int4 ent = list_entry(prm.tile_src + q);
        const int sidx = ent.x, a = X - ent.y, bb = Y - ent.z;
        if (a >= 0 && a <= P && bb >= 0 && bb <= P) {
          const float val = (float)prm.stf[sidx];
          const float *sv = prm.src_vals + (size_t)sidx * 2 * NPE + 2 * (a + bb * N1);
          fx = fmaf(val, sv[0], fx);
          fy = fmaf(val, sv[1], fy);
        }
      }
      const float2 acc = make_float2(fx * d.minv, fy * d.minv);
      if (own)
        SE2P_COLD for (int q = r0; q < r1; q++) {
          const int4 ent = list_entry(prm.tile_rec + q);
          const int r = ent.x, a = X - ent.y, bb = Y - ent.z;
          if (a >= 0 && a <= P && bb >= 0 && bb <= P) {
            float *rb = prm.rbuf_out + ((size_t)r * NPE + a + bb * N1) * 6;
            rb[0] = u.x; rb[1] = u.y; rb[2] = fmaf(half_dt, acc.x, w.x); rb[3] = fmaf(half_dt, acc.y, w.y);
            rb[4] = acc.x; rb[5] = acc.y;
          }
        }
      if (KAHAN) {
        kahan_add(w.x, cw.x, dt * acc.x); kahan_add(w.y, cw.y, dt * acc.y);
        kahan_add(u.x, cu.x, dt * w.x); kahan_add(u.y, cu.y, dt * w.y);
      } else {
        w.x = fmaf(dt, acc.x, w.x); w.y = fmaf(dt, acc.y, w.y);
        u.x = fmaf(dt, w.x, u.x); u.y = fmaf(dt, w.y, u.y);
      }
      if (own) {
        prm.u_out[n] = u;
        prm.w_out[n] = w;
        if (KAHAN) { prm.cu_out[n] = cu; prm.cw_out[n] = cw; }
        if (dp.mode == EF_LAST) prm.a_out[n] = acc;
      }
    }
    sU[i] = u;
    if (KAHAN) sC[i] = cu;
  }
  if (dp.mode == EF_LAST) return;

  // ---- the element forces: one thread per (element, line j)
  const int el = threadIdx.x / N1, j = threadIdx.x - el * N1, ecy = el / TE, ecx = el - ecy * TE;
  const bool active = el < NE && ecx < nex && ecy < ney;
  const int ex = ex0 + ecx, ey = ey0 + ecy;
  const float4 cc = active ? prm.cellc[(size_t)ey * prm.mx + ex] : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();

  // ---- 1. derivatives along row j (registers) and column j (to X1) -----
  float2 gxi[N1];
  const int base = (ecy * P) * RW + ecx * P;
  if (active) {
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      const int stride = dir ? RW : 1, b0 = dir ? base + j : base + j * RW;
      const float2 u0 = sU[b0], c0 = KAHAN ? sC[b0] : make_float2(0.f, 0.f);
      float2 d[N1];
#pragma unroll
      for (int k = 1; k < N1; k++) {
        const float2 uk = sU[b0 + k * stride];
        d[k].x = uk.x - u0.x; d[k].y = uk.y - u0.y;
        if (KAHAN) {
          const float2 ck = sC[b0 + k * stride];
          d[k].x -= (ck.x - c0.x); d[k].y -= (ck.y - c0.y);
        }
      }
#pragma unroll
      for (int q = 0; q < N1; q++) {
        float sx = 0.f, sy = 0.f;
#pragma unroll
        for (int k = 1; k < N1; k++) { sx = fmaf(D[q * N1 + k], d[k].x, sx); sy = fmaf(D[q * N1 + k], d[k].y, sy); }
        if (dir) X1[el * XS + j + q * RS] = make_float2(sx, sy);   // d/deta at (j, q)
        else gxi[q] = make_float2(sx, sy);
      }
    }
  }
  __syncthreads();

  // ---- 2. stress at the row's points; xi divergence to X1; eta fluxes to X2 ---
  if (active) {
    const float lam = cc.x, mu = cc.y, ix = cc.z, iy = cc.w;   // (lam detJ, mu detJ, d xi/dx, d eta/dy)
    const float c11 = fmaf(2.f, mu, lam);
    const float nfj = -W[j];
    float2 Fxi[N1];
#pragma unroll
    for (int q = 0; q < N1; q++) {
      const float2 ge = X1[el * XS + q + j * RS];   // d/deta at (q, j)
      const float e0 = ix * gxi[q].x, e1 = iy * ge.y, e2 = fmaf(ix, gxi[q].y, iy * ge.x);
      const float nf = nfj * W[q];                   // -detJ w_q w_j
      const float fx_ = ix * nf, fy_ = iy * nf;
      const float sxx = fmaf(c11, e0, lam * e1), syy = fmaf(lam, e0, c11 * e1), sxy = mu * e2;
      Fxi[q] = make_float2(fx_ * sxx, fx_ * sxy);
      X2[el * XS + q + j * RS] = make_float2(fy_ * sxy, fy_ * syy);
    }
#pragma unroll
    for (int a = 0; a < N1; a++) {
      float rx = 0.f, ry = 0.f;
#pragma unroll
      for (int q = 0; q < N1; q++) { rx = fmaf(D[q * N1 + a], Fxi[q].x, rx); ry = fmaf(D[q * N1 + a], Fxi[q].y, ry); }
      X1[el * XS + a + j * RS] = make_float2(rx, ry);
    }
  }
  __syncthreads();

  // ---- 3. eta part of the divergence along column j, added to the xi part: the element's forces
  if (active) {
    float2 *ef = static_cast<float2 *>(dp.ef_out) + ((size_t)ey * prm.mx + ex) * NPE;
    float2 fc[N1];
#pragma unroll
    for (int q = 0; q < N1; q++) fc[q] = X2[el * XS + j + q * RS];
#pragma unroll
    for (int bq = 0; bq < N1; bq++) {
      const float2 r = X1[el * XS + j + bq * RS];
      float cx = r.x, cy = r.y;
#pragma unroll
      for (int q = 0; q < N1; q++) { cx = fmaf(D[q * N1 + bq], fc[q].x, cx); cy = fmaf(D[q * N1 + bq], fc[q].y, cy); }
      ef[j + bq * N1] = make_float2(cx, cy);
    }
  }
}

}  // namespace se2p
