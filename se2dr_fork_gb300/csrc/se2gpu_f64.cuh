// se2gpu_f64.cuh -- the explicit step in the reference's FP64 arithmetic, for sm_103a.
//
//   u' = u + dt v + dt^2/2 a,  v* = v + dt/2 a               (se2wave.c:4726-4730)
//   f  = K(u') + sum_s stf_s(t) g_s                           (4733-4739, 1285-1429, 3470-3497)
//   a' = f / M,  v' = v* + dt/2 a'                            (4742-4745)
//
// Bits.  Every product and sum is rounded by itself, in the reference's order.  The
// reference's dense sums over all npe basis functions only add exact zeros outside the
// tensor row and column of a point; restricting each sum to them, in the same order,
// gives the same bits.  A sum that starts at its first term instead of at +0 differs
// only when every term is -0; such a zero can only change the sign of a zero force,
// which plus_zero() restores.
//
// Rate.  What bounds a step is the FP64 pipe (one warp instruction every 16 cycles per
// SM).  Measured on GB300: separately rounded multiplies and adds (two operands) issue
// at 0.528 T/s, fused multiply-adds with three register operands at 0.627 T/s, the
// pipe's full rate.  So a product is issued as fma(a, b, -0) and a sum as
// fma(a, 1, b): both are exact restatements (one rounding of the same real number, and
// x + (-0) = x for every x, zeros included).  The constants 1 and -0 come from memory,
// into registers, because the compiler would turn a visible constant back into the
// two-operand instruction.
//
// No halo.  A step is two passes over different data: the forces of an element need its
// own nodes only, a node needs the forces of its 1, 2 or 4 elements.  A kernel boundary
// between them would leave the FP64 pipe idle during the second, so a launch first
// finishes the previous step at the nodes of its tile (element forces from memory,
// a', v', then the predictor of this step) and then evaluates this step's element
// forces, which it leaves in memory for the next launch.  Only the nodes on tile edges are
// finished twice; no element is evaluated twice, so a tile can be as small as one
// element and small meshes spread over all SMs.  A block of n steps is one START launch
// (from u, v, a), n - 1 MIDDLE launches and one pass over the nodes that forms the last a
// and v.  The element forces (16 (p+1)^2 bytes per element, two buffers) cost memory
// traffic, about 130 B per node-step at degree 4, that a pipe-bound kernel has to spare
// (96 B measured at 1M nodes in 363 us: 4 % of HBM's rate).  The order of a node's
// element sum is ascending, as the reference's VecSetValues(ADD) loop (1417).
//
// Measured on GB300, against one launch per step of 8 x 8 element tiles that also evaluated a
// halo of elements, with two-operand instructions: 1M nodes, degree 4: 560 -> 366 us per step,
// the FP64 pipe 95-96 % active (84 % before), 211 FP64 operations per node (295); 64 x 64
// elements, degree 6: 210 -> 67 us; 8 x 8 elements, degree 2: 29 -> 7 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "se2gpu_f64_launch.h"

namespace se2 {

// Elements per tile and threads, three sizes per degree: (p+1)^2 points per element that fill
// whole warps (the lanes of a last, partly filled warp idle through all of it).  Larger tiles
// finish fewer nodes twice; smaller ones spread a small mesh over more SMs.  f64_launch_step
// chooses.
template <int P, int SIZE> struct F64Tile;
#define SE2_F64_TILE(P, S, TX_, TY_, NT_) \
  template <> struct F64Tile<P, S> { static constexpr int TX = TX_, TY = TY_, NT = NT_; };
SE2_F64_TILE(1, 0, 4, 2, 32) SE2_F64_TILE(1, 1, 8, 4, 128) SE2_F64_TILE(1, 2, 16, 8, 256)
SE2_F64_TILE(2, 0, 3, 1, 32) SE2_F64_TILE(2, 1, 7, 2, 128) SE2_F64_TILE(2, 2, 8, 4, 288)
SE2_F64_TILE(3, 0, 2, 1, 32) SE2_F64_TILE(3, 1, 4, 2, 128) SE2_F64_TILE(3, 2, 4, 4, 256)
SE2_F64_TILE(4, 0, 1, 1, 32) SE2_F64_TILE(4, 1, 5, 1, 128) SE2_F64_TILE(4, 2, 5, 4, 256)
SE2_F64_TILE(5, 0, 1, 1, 64) SE2_F64_TILE(5, 1, 3, 2, 224) SE2_F64_TILE(5, 2, 4, 2, 288)
SE2_F64_TILE(6, 0, 1, 1, 64) SE2_F64_TILE(6, 1, 5, 1, 256) SE2_F64_TILE(6, 2, 5, 3, 256)
SE2_F64_TILE(7, 0, 1, 1, 64) SE2_F64_TILE(7, 1, 2, 1, 128) SE2_F64_TILE(7, 2, 4, 2, 256)
SE2_F64_TILE(8, 0, 1, 1, 96) SE2_F64_TILE(8, 1, 3, 1, 256) SE2_F64_TILE(8, 2, 4, 2, 256)
#undef SE2_F64_TILE

// products and sums on the fused pipe (see above)
struct F64Ops {
  double one, nzero;
  __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, nzero); }
  __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
};
__device__ __forceinline__ F64Ops f64_ops(const double *constants)
{
  const volatile double *c = constants;
  return F64Ops{c[0], c[1]};
}
__device__ __forceinline__ double plus_zero(double x)
{
  return (__double_as_longlong(x) == (long long)0x8000000000000000ULL) ? 0.0 : x;
}

// f / m, correctly rounded, from r = 1/m correctly rounded: two Newton corrections of the
// quotient with exact remainders (Markstein, IBM J. Res. Dev. 34, 1990: with r the
// rounded reciprocal and q faithful, q + r (f - m q) rounds to the quotient; the first
// correction makes q faithful).  The range test keeps every remainder exact; outside
// it, and where r is 0, the division itself.
__device__ __forceinline__ double f64_div(double f, double m, double r)
{
  const int e = (__double2hiint(f) >> 20) & 0x7ff;
  const bool safe = (e > 223 && e < 1823) || f == 0.0;
  if (!safe || r == 0.0) return __ddiv_rn(f, m);
  double q = f * r;
  q = __fma_rn(__fma_rn(-m, q, f), r, q);
  return __fma_rn(__fma_rn(-m, q, f), r, q);
}

// f = sum of the element forces at node (X, Y), ascending element order
template <int P>
__device__ __forceinline__ double2 f64_gather(const double2 *ef, int mx, int my, int X, int Y, const F64Ops &o)
{
  constexpr int N1 = P + 1, NPE = N1 * N1;
  const int ex = X / P, ey = Y / P, ix = X - ex * P, iy = Y - ey * P;
  const bool in_x = ex < mx, in_y = ey < my, lft = ix == 0 && ex > 0, bot = iy == 0 && ey > 0;
  const double2 *own = ef + ((size_t)ey * mx + ex) * NPE + ix + iy * N1;   // (dereferenced only inside the mesh)
  const bool c0 = bot && lft, c1 = bot && in_x, c2 = lft && in_y, c3 = in_x && in_y;
  double2 g0, g1, g2, g3;
  if (c0) g0 = own[-(ptrdiff_t)(mx + 1) * NPE + P + P * N1];
  if (c1) g1 = own[-(ptrdiff_t)mx * NPE + P * N1];
  if (c2) g2 = own[-(ptrdiff_t)NPE + P];
  if (c3) g3 = own[0];
  double2 f = make_double2(0.0, 0.0);
  if (c0) f = g0;
  if (c1) {
    if (c0) { f.x = o.add(f.x, g1.x); f.y = o.add(f.y, g1.y); }
    else f = g1;
  }
  if (c2) {
    if (c0 || c1) { f.x = o.add(f.x, g2.x); f.y = o.add(f.y, g2.y); }
    else f = g2;
  }
  if (c3) {
    if (c0 || c1 || c2) { f.x = o.add(f.x, g3.x); f.y = o.add(f.y, g3.y); }
    else f = g3;
  }
  return make_double2(plus_zero(f.x), plus_zero(f.y));
}

// a' and v' of node (X, Y) from v* and the element forces of the step
template <int P>
__device__ __forceinline__ void f64_finish(const F64Params &q, const double2 *ef, const double2 vs, int X, int Y,
                                           const F64Ops &o, double2 &v, double2 &a)
{
  constexpr int N1 = P + 1, NPE = N1 * N1;
  const size_t n = (size_t)Y * q.nx_g + X;
  const double m = q.mass[n], r = q.rmass[n];
  double2 f = f64_gather<P>(ef, q.mx, q.my, X, Y, o);
  // source injection: g = sum_s stf_s g_s (from +0), then f + 1.0 g; a node without sources
  // adds +0, which plus_zero has done
  double gx = 0.0, gy = 0.0;
  bool any = false;
  for (int s = 0; s < q.nsrc; s++) {
    const int2 e = q.src_xy[s];
    const int ia = X - e.x, ib = Y - e.y;
    if (ia >= 0 && ia <= P && ib >= 0 && ib <= P) {
      const double val = q.stf[s];
      const double *sv = q.src_vals + (size_t)s * 2 * NPE + 2 * (ia + ib * N1);
      gx = __dadd_rn(gx, __dmul_rn(val, sv[0]));
      gy = __dadd_rn(gy, __dmul_rn(val, sv[1]));
      any = true;
    }
  }
  if (any) { f.x = __dadd_rn(f.x, gx); f.y = __dadd_rn(f.y, gy); }
  a.x = f64_div(f.x, m, r);
  a.y = f64_div(f.y, m, r);
  v.x = o.add(vs.x, o.mul(q.c_v, a.x));
  v.y = o.add(vs.y, o.mul(q.c_v, a.y));
}

// one warp per receiver (se2wave.c:2908-2962): u, v, a at its node, and curl(v) from the row
// and column of its element through the node.  Lanes 0..P take the column, P+1..2P+1 the
// row; the sums run in ascending order.
template <int P>
__device__ void f64_sample(const F64Params &q, int first, int stride, const F64Ops &o)
{
  constexpr int N1 = P + 1;
  const int lane = threadIdx.x & 31;
  for (int r = first; r < q.nrec; r += stride) {
    const int eid = q.rec_elem[r], g = q.rec_gll[r];
    const int ex = eid % q.mx, ey = eid / q.mx, ga = g % N1, gb = g / N1;
    const bool col = lane < N1, row = !col && lane < 2 * N1;
    const int k = col ? lane : row ? lane - N1 : 0;
    double pr = 0.0;
    if (col || row) {
      const int X = ex * P + (col ? ga : k), Y = ey * P + (col ? k : gb);
      const size_t n = (size_t)Y * q.nx_g + X;
      double2 v = q.v_in[n], a;
      if (q.mode == F64_MIDDLE) f64_finish<P>(q, q.ef_in, q.v_in[n], X, Y, o, v, a);
      else a = q.a_in[n];
      if (col && k == gb) {
        const double2 u = q.u_in[n];
        double *t = q.trace_row + 7 * r;
        t[0] = u.x; t[1] = u.y; t[2] = v.x; t[3] = v.y; t[4] = a.x; t[5] = a.y;
      }
      pr = col ? __dmul_rn(__dmul_rn(q.iJ11d[ey], q.Dd[gb * N1 + k]), v.x)
               : __dmul_rn(__dmul_rn(q.iJ00d[ex], q.Dd[ga * N1 + k]), v.y);
    }
    double dvxdy = 0.0, dvydx = 0.0;
    for (int i = 0; i < N1; i++) dvxdy = __dadd_rn(dvxdy, __shfl_sync(0xffffffffu, pr, i));
    for (int i = 0; i < N1; i++) dvydx = __dadd_rn(dvydx, __shfl_sync(0xffffffffu, pr, N1 + i));
    if (lane == 0) q.trace_row[7 * r + 6] = __dadd_rn(dvydx, -dvxdy);
  }
}

// term t (0 .. 2P) of a sum that takes the column entries before `at`, the row, and the
// column entries after `at`; row[] holds the diagonal's combined term
template <int P>
__device__ __forceinline__ double f64_term(int t, int at, const double (&col)[P + 1], const double (&row)[P + 1])
{
  double v = 0.0;
#pragma unroll
  for (int c = (t > P ? t - P : 0); c <= (t < P ? t : P); c++)
    if (at == c) v = row[t - c];
  if (t < P && t < at) v = col[t < P ? t : 0];
  if (t > P && t - P > at) v = col[t > P ? t - P : 0];
  return v;
}

// (programmatic dependent launch: a launch may begin while the one before it drains; only the
// tables that no launch writes are read ahead of the wait)
template <int P, int SIZE>
__global__ void __launch_bounds__(F64Tile<P, SIZE>::NT, 512 / F64Tile<P, SIZE>::NT) f64_step(const F64Params q)
{
  typedef F64Tile<P, SIZE> T;
  constexpr int TX = T::TX, TY = T::TY, NT = T::NT, N1 = P + 1, NPE = N1 * N1;
  constexpr int RW = TX * P + 1, RH = TY * P + 1, ITEMS = TX * TY * NPE;
  __shared__ double2 sU[RW * RH];
  __shared__ double sS[ITEMS * 3];          // (sxx, sxy, syy) per point
  __shared__ double sNf[ITEMS];             // -(detJ w_q) per point
  __shared__ double sDx[TX * NPE], sDy[TY * NPE], sDet[TX * TY];
  const F64Ops o = f64_ops(q.constants);

  if ((int)blockIdx.x >= q.ntiles) {
    constexpr int WARPS = NT / 32;
    cudaGridDependencySynchronize();
    f64_sample<P>(q, ((int)blockIdx.x - q.ntiles) * WARPS + (threadIdx.x >> 5), q.nsamp * WARPS, o);
    return;
  }
  const int tx = blockIdx.x % q.ntx, ty = blockIdx.x / q.ntx;
  const int ex0 = tx * TX, ey0 = ty * TY, nex = min(TX, q.mx - ex0), ney = min(TY, q.my - ey0);
  const int X0 = ex0 * P, Y0 = ey0 * P;
  for (int i = threadIdx.x; i < nex * NPE; i += NT) sDx[i] = q.Dx[(size_t)ex0 * NPE + i];
  for (int i = threadIdx.x; i < ney * NPE; i += NT) sDy[i] = q.Dy[(size_t)ey0 * NPE + i];
  for (int i = threadIdx.x; i < TX * TY; i += NT)
    if (i % TX < nex && i / TX < ney) sDet[i] = o.mul(q.J00[ex0 + i % TX], q.J11[ey0 + i / TX]);
  cudaGridDependencySynchronize();

  // ---- finish the previous step and predict this one at the tile's nodes; a node line
  // shared with the next tile belongs to that one, which writes it
  const int own_w = nex * P + (ex0 + nex == q.mx ? 1 : 0), own_h = ney * P + (ey0 + ney == q.my ? 1 : 0);
  for (int i = threadIdx.x; i < RW * RH; i += NT) {
    const int ry = i / RW, rx = i - ry * RW;
    if (rx > nex * P || ry > ney * P) continue;
    const int X = X0 + rx, Y = Y0 + ry;
    const size_t n = (size_t)Y * q.nx_g + X;
    double2 u = q.u_in[n];
    if (q.mode != F64_FORCE) {
      double2 v = q.v_in[n], a;
      if (q.mode == F64_MIDDLE) {
        const double2 vs = v;
        f64_finish<P>(q, q.ef_in, vs, X, Y, o, v, a);
      } else {
        a = q.a_in[n];
      }
      // VecAXPY(u,dt,v); VecAXPY(u,0.5*dt*dt,a); VecAXPY(v,0.5*dt,a)
      u.x = o.add(o.add(u.x, o.mul(q.c_dt, v.x)), o.mul(q.c_u, a.x));
      u.y = o.add(o.add(u.y, o.mul(q.c_dt, v.y)), o.mul(q.c_u, a.y));
      if (rx < own_w && ry < own_h) {
        v.x = o.add(v.x, o.mul(q.c_v, a.x));
        v.y = o.add(v.y, o.mul(q.c_v, a.y));
        q.u_out[n] = u;
        q.v_out[n] = v;
      }
    }
    sU[i] = u;
  }
  __syncthreads();

  // ---- strain and Hooke stress at every GLL point.  The FP64 pipe leaves some 60 issue
  // slots of other instructions free per FP64 instruction, so the ordered shear sum is
  // taken with selects (the same instructions for every point) instead of branches.
  for (int it = threadIdx.x; it < ITEMS; it += NT) {
    const int el = it / NPE, p = it - el * NPE, ecy = el / TX, ecx = el - ecy * TX;
    if (ecx >= nex || ecy >= ney) continue;
    const int qj = p / N1, qi = p - qj * N1;
    const double2 *ue = sU + (ecy * P) * RW + ecx * P;
    const size_t cell = (size_t)(ey0 + ecy) * q.mx + ex0 + ecx;
    const double lam = q.lam[cell], mu = q.mu[cell];
    const double *dx = sDx + ecx * NPE + qi * N1;   // dN/dx of basis (ia, qj) at the point
    const double *dy = sDy + ecy * NPE + qj * N1;   // dN/dy of basis (qi, ib)
    double e0 = 0.0, e1 = 0.0, row[N1], col[N1], rd = 0.0, cd = 0.0;
#pragma unroll
    for (int k = 0; k < N1; k++) {
      const double2 ur = ue[qj * RW + k], uc = ue[k * RW + qi];
      const double dxk = dx[k], dyk = dy[k];
      const double px = o.mul(dxk, ur.x), py = o.mul(dyk, uc.y);
      e0 = k ? o.add(e0, px) : px;
      e1 = k ? o.add(e1, py) : py;
      row[k] = o.mul(dxk, ur.y);
      col[k] = o.mul(dyk, uc.x);
      if (k == qi) rd = row[k];
      if (k == qj) cd = col[k];
    }
    const double diag = o.add(rd, cd);
#pragma unroll
    for (int k = 0; k < N1; k++)
      if (k == qi) row[k] = diag;
    // shear strain: basis index ascending = column below, row, column above
    double e2 = f64_term<P>(0, qj, col, row);
#pragma unroll
    for (int t = 1; t <= 2 * P; t++) e2 = o.add(e2, f64_term<P>(t, qj, col, row));
    const double c11 = __fma_rn(2.0, mu, lam);   // 2 mu is exact
    sS[3 * it] = o.add(o.mul(c11, e0), o.mul(lam, e1));
    sS[3 * it + 1] = o.mul(mu, e2);
    sS[3 * it + 2] = o.add(o.mul(lam, e0), o.mul(c11, e1));
    sNf[it] = -o.mul(sDet[el], q.wq[p]);
  }
  __syncthreads();

  if (q.trigger) cudaTriggerProgrammaticLaunchCompletion();
  // ---- weak divergence at the element's nodes: quadrature points ascending = column below
  // the node's row, the row, column above
  for (int it = threadIdx.x; it < ITEMS; it += NT) {
    const int el = it / NPE, p = it - el * NPE, ecy = el / TX, ecx = el - ecy * TX;
    if (ecx >= nex || ecy >= ney) continue;
    const int b = p / N1, a = p - b * N1;
    const double *S = sS + 3 * el * NPE, *nf = sNf + el * NPE;
    const double *dx = sDx + ecx * NPE + a, *dy = sDy + ecy * NPE + b;
    double rx[N1], ry[N1], cx[N1], cy[N1], drx = 0.0, dry = 0.0, dcx = 0.0, dcy = 0.0;
#pragma unroll
    for (int k = 0; k < N1; k++) {
      const double *Sr = S + 3 * (k + b * N1), *Sc = S + 3 * (a + k * N1);
      const double dNx = dx[k * N1], dNy = dy[k * N1];
      rx[k] = o.mul(dNx, Sr[0]);
      ry[k] = o.mul(dNx, Sr[1]);
      cx[k] = o.mul(dNy, Sc[1]);
      cy[k] = o.mul(dNy, Sc[2]);
      if (k == a) { drx = rx[k]; dry = ry[k]; }
      if (k == b) { dcx = cx[k]; dcy = cy[k]; }
    }
    const double dgx = o.add(drx, dcx), dgy = o.add(dcy, dry);
#pragma unroll
    for (int k = 0; k < N1; k++)
      if (k == a) { rx[k] = dgx; ry[k] = dgy; }
    double gx = 0.0, gy = 0.0;
#pragma unroll
    for (int t = 0; t <= 2 * P; t++) {
      const int pt = (t < b) ? a + t * N1 : (t <= b + P) ? (t - b) + b * N1 : a + (t - P) * N1;
      const double w = nf[pt];
      const double vx = o.mul(w, f64_term<P>(t, b, cx, rx)), vy = o.mul(w, f64_term<P>(t, b, cy, ry));
      gx = t ? o.add(gx, vx) : vx;
      gy = t ? o.add(gy, vy) : vy;
    }
    q.ef_out[((size_t)(ey0 + ecy) * q.mx + ex0 + ecx) * NPE + p] = make_double2(gx, gy);
  }
}

// the last step of a block: v' and a' at every node (v in place, a to a_out)
template <int P>
__global__ void __launch_bounds__(256) f64_last(const F64Params q, double2 *v, double2 *a_out)
{
  const F64Ops o = f64_ops(q.constants);
  cudaGridDependencySynchronize();
  for (int Y = blockIdx.y; Y < q.ny_g; Y += gridDim.y) {
    const int X = blockIdx.x * blockDim.x + threadIdx.x;
    if (X >= q.nx_g) return;
    const size_t n = (size_t)Y * q.nx_g + X;
    double2 vn, an;
    f64_finish<P>(q, q.ef_in, v[n], X, Y, o, vn, an);
    v[n] = vn;
    a_out[n] = an;
  }
}

// the internal force at every node from the element forces
template <int P>
__global__ void __launch_bounds__(256) f64_force(const F64Params q, double2 *f_out)
{
  const F64Ops o = f64_ops(q.constants);
  cudaGridDependencySynchronize();
  for (int Y = blockIdx.y; Y < q.ny_g; Y += gridDim.y) {
    const int X = blockIdx.x * blockDim.x + threadIdx.x;
    if (X >= q.nx_g) return;
    f_out[(size_t)Y * q.nx_g + X] = f64_gather<P>(q.ef_in, q.mx, q.my, X, Y, o);
  }
}

// receiver rows of the state u, v, a
template <int P>
__global__ void __launch_bounds__(128) f64_record(const F64Params q)
{
  f64_sample<P>(q, blockIdx.x * 4 + (threadIdx.x >> 5), gridDim.x * 4, f64_ops(q.constants));
}

// 1/M rounded to nearest, 0 where f64_div must divide
__global__ void f64_reciprocal(const double *mass, double *r, size_t n)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int e = (__double2hiint(mass[i]) >> 20) & 0x7ff;
    r[i] = (e > 923 && e < 1123) ? __drcp_rn(mass[i]) : 0.0;
  }
}

}  // namespace se2
