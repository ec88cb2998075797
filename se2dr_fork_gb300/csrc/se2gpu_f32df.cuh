// se2gpu_f32df.cuh -- the step in two-float arithmetic, for sm_103a.
//
// The same leapfrog as se2gpu_persist.cuh (state u, w with their low parts stored as Kahan terms:
// value = hi - c) with every value of a step an unevaluated sum of two floats.  What bounds it on
// large meshes is instruction issue (77 % of the issue slots busy, memory a quarter), so
// no element is evaluated twice: as in the FP64 step (se2gpu_f64.cuh) a launch finishes the previous
// step at the nodes of its tile, from the element forces in memory, and then leaves this step's
// element forces there.  Only the nodes on tile edges are finished twice, where a halo of elements
// cost a third of the element work.  The forces (16 (p+1)^2 bytes per element, two buffers) add
// about 50 B per node and step at degree 4.  3.53M nodes, degree 4, 6 steps: 1313 -> 1169 us; degree 7
// at 2.5M nodes 304 -> 176 us a step, 20000 nodes 19.4 -> 11.9 (every size: se2gpu_f32df_launch.h).
//
// A block of n steps: one EF_START launch (element forces of the state), n - 1 EF_MIDDLE
// launches, and EF_LAST, which finishes the last step at every node and stores its a (df_last).
#pragma once
#include "se2gpu_persist.cuh"
#include "se2gpu_f32df_launch.h"

namespace se2p {

// nodes of the region a tile of TE x TE elements touches, and its exchange rows
template <int P, int TE>
struct DfGeo {
  static constexpr int N1 = P + 1, NPE = N1 * N1, RW = TE * P + 1, NE = TE * TE;
  // (the row pitch and the element pitch put the points that a warp touches, along rows and along
  // columns, on different banks)
  static constexpr int RP = df_row_pitch(P), XS = df_elem_pitch(P);
  static constexpr size_t SMEM = sizeof(float4) * ((size_t)RW * RW + 2 * (size_t)NE * XS);
};

// what a node of the step to finish reads: its state and the forces of the up to four elements
// around it, in ascending element order.  Loaded one node ahead of its use: the loads of a node
// are independent, so a thread waits once per node, and ahead of that wait it has arithmetic left
struct DfNode {
  float2 u, cu, w, cw;
  float minv_h, minv_l;
  float4 g[4];
};

template <int P>
__device__ __forceinline__ void df_load(const EfParams &dp, int X, int Y, DfNode &d)
{
  constexpr int N1 = P + 1, NPE = N1 * N1;
  const Params &prm = dp.p;
  const size_t n = (size_t)Y * prm.pitch + X;
  d.u = dp.u_in[n];
  d.cu = dp.cu_in[n];
  if (dp.mode == EF_START) return;
  d.w = dp.w_in[n];
  d.cw = dp.cw_in[n];
  d.minv_h = prm.minv[n];
  d.minv_l = prm.minv[(size_t)prm.ny_g * prm.pitch + n];
  const NodePos<P> c(prm.mx, prm.my, X, Y);
  const float4 *ef = static_cast<const float4 *>(dp.ef_in) + ((ptrdiff_t)c.ey * prm.mx + c.ex) * NPE + c.ix + c.iy * N1;
  if (c.bot && c.lft) d.g[0] = ef[-(ptrdiff_t)(prm.mx + 1) * NPE + P + P * N1];
  if (c.bot && c.in_x) d.g[1] = ef[-(ptrdiff_t)prm.mx * NPE + P * N1];
  if (c.lft && c.in_y) d.g[2] = ef[-(ptrdiff_t)NPE + P];
  if (c.in_x && c.in_y) d.g[3] = ef[0];
}

// the step of node (X, Y): a, then w and u, in the state's arithmetic; receivers' values where this
// thread owns the node.  bnd: source and receiver list bounds of the node's tile
struct DfStep {
  tf ax, ay, wx, wy, ux, uy;
};
template <int P>
__device__ __forceinline__ DfStep df_finish(const EfParams &dp, const DfNode &d, int X, int Y, const int4 bnd, bool own)
{
  constexpr int N1 = P + 1, NPE = N1 * N1;
  const Params &prm = dp.p;
  const tf dt{prm.dt, prm.dt_lo}, hdt{prm.half_dt, prm.half_dt_lo};
  const float *src_lo = prm.src_vals + (size_t)prm.nsrc * 2 * NPE;
  tf fx{0.f, 0.f}, fy{0.f, 0.f};
  {
    const NodePos<P> c(prm.mx, prm.my, X, Y);
    const bool have[4] = {c.bot && c.lft, c.bot && c.in_x, c.lft && c.in_y, c.in_x && c.in_y};
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (have[k]) {
        fx = tf_add(fx, tf{d.g[k].x, d.g[k].z});
        fy = tf_add(fy, tf{d.g[k].y, d.g[k].w});
      }
  }
  SE2P_COLD for (int q = bnd.x; q < bnd.y; q++) {
    const int4 ent = list_entry(prm.tile_src + q);
    const int sidx = ent.x, a = X - ent.y, bb = Y - ent.z;
    if (a >= 0 && a <= P && bb >= 0 && bb <= P) {
      const tf val = tf_from_double(prm.stf[sidx]);
      const size_t vi = (size_t)sidx * 2 * NPE + 2 * (a + bb * N1);
      fx = tf_add(fx, tf_mul(val, tf{prm.src_vals[vi], src_lo[vi]}));
      fy = tf_add(fy, tf_mul(val, tf{prm.src_vals[vi + 1], src_lo[vi + 1]}));
    }
  }
  const tf minv{d.minv_h, d.minv_l};
  const tf ax = tf_mul(fx, minv), ay = tf_mul(fy, minv);
  const tf ux{d.u.x, -d.cu.x}, uy{d.u.y, -d.cu.y}, wx{d.w.x, -d.cw.x}, wy{d.w.y, -d.cw.y};
  if (own)
    SE2P_COLD for (int q = bnd.z; q < bnd.w; q++) {
      const int4 ent = list_entry(prm.tile_rec + q);
      const int r = ent.x, a = X - ent.y, bb = Y - ent.z;
      if (a >= 0 && a <= P && bb >= 0 && bb <= P) {
        float *rb = prm.rbuf_out + ((size_t)r * NPE + a + bb * N1) * 12;
        const tf vx = tf_add(wx, tf_mul(hdt, ax)), vy = tf_add(wy, tf_mul(hdt, ay));
        const tf uxn = tf_norm(ux), uyn = tf_norm(uy);
        rb[0] = uxn.h; rb[1] = uyn.h; rb[2] = vx.h; rb[3] = vy.h; rb[4] = ax.h; rb[5] = ay.h;
        rb[6] = uxn.l; rb[7] = uyn.l; rb[8] = vx.l; rb[9] = vy.l; rb[10] = ax.l; rb[11] = ay.l;
      }
    }
  const tf wxn = tf_add(wx, tf_mul(dt, ax)), wyn = tf_add(wy, tf_mul(dt, ay));
  return DfStep{ax, ay, wxn, wyn, tf_add(ux, tf_mul(dt, wxn)), tf_add(uy, tf_mul(dt, wyn))};
}
__device__ __forceinline__ void df_store(const EfParams &dp, size_t n, const DfStep &r)
{
  dp.p.u_out[n] = make_float2(r.ux.h, r.uy.h);
  dp.p.w_out[n] = make_float2(r.wx.h, r.wy.h);
  dp.p.cu_out[n] = make_float2(-r.ux.l, -r.uy.l);
  dp.p.cw_out[n] = make_float2(-r.wx.l, -r.wy.l);
}

// EF_LAST: the last step of a block at every node, and its a: one thread per node, each read once,
// whatever the tiles (tile_nodes: nodes of a tile along an edge, for the lists).  It moves memory
// only.  Walking the element kernel's tiles (a node of a CTA's region after the other, nodes on tile
// edges idle) took 81 us at 2.5M nodes, degree 4, which made a block of a single step slower than
// the step with a halo (160 -> 180 us); this takes 40 (single step 139).
constexpr int DF_LX = 32, DF_LY = 8;   // nodes of a CTA along x and y
template <int P>
__global__ void __launch_bounds__(DF_LX * DF_LY) df_last(const EfParams dp, int tile_nodes, int nbx, int nblocks)
{
  const Params &prm = dp.p;
  cudaGridDependencySynchronize();
  if ((int)blockIdx.x >= nblocks) {   // (one more CTA: the receivers of the step before)
    sample_rows<P, true>(prm, prm.rbuf_in, prm.trace_row);
    return;
  }
  const int by = blockIdx.x / nbx, bx = blockIdx.x - by * nbx;
  const int X = bx * DF_LX + threadIdx.x % DF_LX, Y = by * DF_LY + threadIdx.x / DF_LX;
  if (X >= prm.nx_g || Y >= prm.ny_g) return;
  DfNode d;
  df_load<P>(dp, X, Y, d);
  const int nty = prm.ntiles / prm.ntx;
  const int tx = min(X / tile_nodes, prm.ntx - 1), ty = min(Y / tile_nodes, nty - 1);
  const DfStep r = df_finish<P>(dp, d, X, Y, prm.tile_bounds[ty * prm.ntx + tx], true);
  const size_t n = (size_t)Y * prm.pitch + X;
  df_store(dp, n, r);
  prm.a_out[n] = make_float2(r.ax.h, r.ay.h);
  prm.a_out[(size_t)prm.ny_g * prm.pitch + n] = make_float2(r.ax.l, r.ay.l);   // low parts after the high parts
}

template <int P, int TE, int NT>
__global__ void __launch_bounds__(NT, df_min_blocks(P, TE, NT)) df_step(const EfParams dp)
{
  typedef DfGeo<P, TE> G;
  constexpr int N1 = G::N1, NPE = G::NPE, RW = G::RW, RP = G::RP, XS = G::XS;
  const Params &prm = dp.p;
  const float *Dh = c_D[P - 1], *Dl = c_Dl[P - 1];
  extern __shared__ __align__(128) unsigned char smem[];
  float4 *sU = reinterpret_cast<float4 *>(smem);   // (u.x, u.y, c.x, c.y)
  float4 *X1 = sU + RW * RW, *X2 = X1 + G::NE * XS;
  cudaGridDependencySynchronize();
  if ((int)blockIdx.x >= prm.ntiles) {   // (one more CTA: the receivers of the step before)
    if (prm.record) sample_rows<P, true>(prm, prm.rbuf_in, prm.trace_row);
    return;
  }
  const int ty = blockIdx.x / prm.ntx, tx = blockIdx.x - ty * prm.ntx;
  const int ex0 = tx * TE, ey0 = ty * TE, nex = min(TE, prm.mx - ex0), ney = min(TE, prm.my - ey0);
  const int X0 = ex0 * P, Y0 = ey0 * P;

  // ---- the tile's nodes: finish the previous step (a node line shared with the next tile belongs to
  // that one, which writes it)
  const int own_w = nex * P + (ex0 + nex == prm.mx ? 1 : 0), own_h = ney * P + (ey0 + ney == prm.my ? 1 : 0);
  const int4 bnd = prm.tile_bounds[blockIdx.x];
  auto load = [&](int i, DfNode &d) {
    const int ry = i / RW, rx = i - ry * RW;
    if (i < RW * RW && rx <= nex * P && ry <= ney * P) df_load<P>(dp, X0 + rx, Y0 + ry, d);
  };
  DfNode next;
  load(threadIdx.x, next);
#pragma unroll 1
  for (int i = threadIdx.x; i < RW * RW; i += NT) {
    const DfNode d = next;
    load(i + NT, next);
    const int ry = i / RW, rx = i - ry * RW;
    if (rx > nex * P || ry > ney * P) continue;
    if (dp.mode == EF_START) {
      sU[i] = make_float4(d.u.x, d.u.y, d.cu.x, d.cu.y);
      continue;
    }
    const bool own = rx < own_w && ry < own_h;
    const DfStep r = df_finish<P>(dp, d, X0 + rx, Y0 + ry, bnd, own);
    sU[i] = make_float4(r.ux.h, r.uy.h, -r.ux.l, -r.uy.l);
    if (own) df_store(dp, (size_t)(Y0 + ry) * prm.pitch + X0 + rx, r);
  }

  // ---- the element forces: one thread per (element, line j)
  const int el = threadIdx.x / N1, j = threadIdx.x - el * N1, ecy = el / TE, ecx = el - ecy * TE;
  const bool active = el < G::NE && ecx < nex && ecy < ney;
  const int ex = ex0 + ecx, ey = ey0 + ecy;
  const size_t ncell = (size_t)prm.mx * prm.my;
  tf lam{0.f, 0.f}, mu{0.f, 0.f}, ix{0.f, 0.f}, iy{0.f, 0.f}, detJ{0.f, 0.f};
  if (active) {
    const size_t cell = (size_t)ey * prm.mx + ex;
    lam = tf{prm.lam[cell], prm.lam[ncell + cell]};
    mu = tf{prm.mu[cell], prm.mu[ncell + cell]};
    ix = tf{prm.iJ00[ex], prm.iJ00[prm.mx + ex]};
    iy = tf{prm.iJ11[ey], prm.iJ11[prm.my + ey]};
    detJ = tf_mul(tf{prm.J00[ex], prm.J00[prm.mx + ex]}, tf{prm.J11[ey], prm.J11[prm.my + ey]});
  }
  __syncthreads();

  // 1. derivatives along row j and column j (to X1), of the displacement relative to the line's
  // first node: (u_k - u_0) + (c_0 - c_k) with the first difference split exactly by TwoSum
  // Next to issue, the fetch of its instructions bounds this part: the loops over directions and
  // points are rolled (what they index goes through the thread's own exchange rows), those over
  // outputs too from degree 5 on, three at a time (degree 4, 2.5M nodes: 173 -> 159 us a step, waits for
  // instructions 1.45 -> 1.05 cycles per issue, 2.0 of 8.7 with the 28 warps that now fit; outputs rolled
  // at degree 5 180 -> 162, at degree 4 159 -> 161).
  constexpr int DU = P >= 5 ? 3 : N1;
  const int base = (ecy * P) * RW + ecx * P;
  if (active) {
#pragma unroll 1
    for (int dir = 0; dir < 2; dir++) {
      const int stride = dir ? RW : 1, b0 = dir ? base + j : base + j * RW;
      // d/dxi at (q, j) to X2, read back by this thread alone; d/deta at (j, q) to X1
      float4 *xo = dir ? X1 + el * XS + j : X2 + el * XS + j * RP;
      const int so = dir ? RP : 1;
      const float4 u0 = sU[b0];   // (u.x, u.y, c.x, c.y)
      tf dx[N1], dy[N1];
#pragma unroll
      for (int k = 1; k < N1; k++) {
        const float4 uk = sU[b0 + k * stride];
        dx[k] = tf_two_sum(uk.x, -u0.x);
        dx[k].l = __fsub_rn(dx[k].l, __fsub_rn(uk.z, u0.z));
        dy[k] = tf_two_sum(uk.y, -u0.y);
        dy[k].l = __fsub_rn(dy[k].l, __fsub_rn(uk.w, u0.w));
      }
#pragma unroll DU
      for (int q = 0; q < N1; q++) {
        tf sx{0.f, 0.f}, sy{0.f, 0.f};
#pragma unroll
        for (int k = 1; k < N1; k++) {
          tf_dot(sx, Dh[q * N1 + k], Dl[q * N1 + k], dx[k]);
          tf_dot(sy, Dh[q * N1 + k], Dl[q * N1 + k], dy[k]);
        }
        sx = tf_norm(sx);
        sy = tf_norm(sy);
        const float4 g = make_float4(sx.h, sy.h, sx.l, sy.l);
        xo[q * so] = g;
      }
    }
  }
  __syncthreads();

  // ---- 2. stress at the row's points: the xi fluxes take the place of the eta derivatives, which
  // this thread alone reads, the eta fluxes that of the xi derivatives; xi divergence
  if (active) {
    const tf c11 = tf_add(tf_add(mu, mu), lam);
    const tf nfj = tf_neg(tf_mul(detJ, tf{c_w[P - 1][j], c_wl[P - 1][j]}));
#pragma unroll 1
    for (int q = 0; q < N1; q++) {
      const int at = el * XS + q + j * RP;
      const float4 g4 = X1[at], x4 = X2[at];   // d/deta and d/dxi at (q, j)
      const tf gx{x4.x, x4.z}, gy{x4.y, x4.w};
      const tf gex{g4.x, g4.z}, gey{g4.y, g4.w};
      const tf e0 = tf_mul(ix, gx), e1 = tf_mul(iy, gey);
      const tf e2 = tf_add(tf_mul(ix, gy), tf_mul(iy, gex));
      const tf nf = tf_mul(nfj, tf{c_w[P - 1][q], c_wl[P - 1][q]});   // -detJ w_q w_j
      const tf fx_ = tf_mul(ix, nf), fy_ = tf_mul(iy, nf);
      const tf sxx = tf_add(tf_mul(c11, e0), tf_mul(lam, e1));
      const tf syy = tf_add(tf_mul(lam, e0), tf_mul(c11, e1));
      const tf sxy = tf_mul(mu, e2);
      const tf Fxq = tf_mul(fx_, sxx), Fyq = tf_mul(fx_, sxy);
      const tf hx = tf_mul(fy_, sxy), hy = tf_mul(fy_, syy);
      X1[at] = make_float4(Fxq.h, Fyq.h, Fxq.l, Fyq.l);
      X2[at] = make_float4(hx.h, hy.h, hx.l, hy.l);
    }
    tf Fx[N1], Fy[N1];
#pragma unroll
    for (int q = 0; q < N1; q++) {
      const float4 f4 = X1[el * XS + q + j * RP];
      Fx[q] = tf{f4.x, f4.z};
      Fy[q] = tf{f4.y, f4.w};
    }
    // xi part of the divergence for the row's nodes, to X1
#pragma unroll DU
    for (int a = 0; a < N1; a++) {
      tf rx{0.f, 0.f}, ry{0.f, 0.f};
#pragma unroll
      for (int q = 0; q < N1; q++) {
        tf_dot(rx, Dh[q * N1 + a], Dl[q * N1 + a], Fx[q]);
        tf_dot(ry, Dh[q * N1 + a], Dl[q * N1 + a], Fy[q]);
      }
      rx = tf_norm(rx);
      ry = tf_norm(ry);
      X1[el * XS + a + j * RP] = make_float4(rx.h, ry.h, rx.l, ry.l);
    }
  }
  __syncthreads();

  // ---- 3. eta part of the divergence along column j, added to the xi part: the element's forces
  if (active) {
    float4 *ef = static_cast<float4 *>(dp.ef_out) + ((size_t)ey * prm.mx + ex) * NPE;
    tf fcx[N1], fcy[N1];
#pragma unroll
    for (int q = 0; q < N1; q++) {
      const float4 f4 = X2[el * XS + j + q * RP];
      fcx[q] = tf{f4.x, f4.z};
      fcy[q] = tf{f4.y, f4.w};
    }
#pragma unroll DU
    for (int bq = 0; bq < N1; bq++) {
      const float4 r = X1[el * XS + j + bq * RP];
      tf cx{r.x, r.z}, cy{r.y, r.w};
#pragma unroll
      for (int q = 0; q < N1; q++) {
        tf_dot(cx, Dh[q * N1 + bq], Dl[q * N1 + bq], fcx[q]);
        tf_dot(cy, Dh[q * N1 + bq], Dl[q * N1 + bq], fcy[q]);
      }
      cx = tf_norm(cx);
      cy = tf_norm(cy);
      ef[j + bq * N1] = make_float4(cx.h, cy.h, cx.l, cy.l);
    }
  }
}

}  // namespace se2p
