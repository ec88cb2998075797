// se2nn_rows.cuh -- the surrogate network's layers as fused kernels, for sm_103a.
//
// A Fourier layer is five contractions around one activation-sized array.  Run as one GEMM
// launch each, every contraction moves that array through memory (67 MB at batch 32) for
// a K of 32 to 128, so what bounds them is memory traffic and launch latency, not the tensor
// pipe.  Fused along the image row -- the unit on which both x transforms and the 1x1
// convolution act -- a layer reads and writes it once:
//
//   row_kernel    one image row (nx pixels x W channels) at a time: the inverse x transform of
//                 the layer's spectrum row, the 1x1 convolution, bias, GELU, and the forward
//                 x transform of the result for the next layer.  Backward: the adjoint of the
//                 same chain with GELU' of the stored pre-activation.
//   y_analysis    per sample: the forward y transform, stored mode-major
//   mode_mix      per mode: the complex channel mixing from the two real weight matrices
//   mode_grad     per mode: the adjoint of the mixing and both weight gradients
//   y_synthesis   per sample: the inverse y transform
//
// Numbers.  Every contraction accumulates in FP32 over k in ascending steps of 16
// (mma.m16n8k16, products of zero padding adding exact zeros), and every array that the
// unfused kernels store in BF16 is rounded to BF16 at the same place, so the results
// are the same bits as the GEMM kernels' (tests/test_nn_fused.py).
//
// Used for W = 16, 32, 48, 64, nx <= 128 a multiple of 16, ny <= 128 a multiple of 8 and up to
// 16 modes (se2nn.cu, fused_ok); other shapes run the GEMM kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "se2nn_gemm.cuh"

namespace nnk {

constexpr int RT = 256;                  // threads of the row kernels
constexpr int RK = 32;                   // x modes (re, im) padded to two k steps
constexpr int RNX = 128, RNY = 128, RM = 16, RREC = 128;   // largest row, column, modes, receivers

template <int LEFT> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// asynchronous copy of rows x cols (a multiple of 8) elements into shared memory.  COLS: the row
// length where it is known (the index then needs no division, a third of the small kernels'
// instructions otherwise)
template <int COLS = 0>
__device__ __forceinline__ void copy_tile(bf16 *s, int lds, const bf16 *g, long ldg, int rows, int cols, int nt)
{
  const int per = (COLS ? COLS : cols) / 8;
  for (int e = threadIdx.x; e < rows * per; e += nt) {
    const int r = e / per, c = (e - r * per) * 8;
    cp_async16(smem_addr(s + r * lds + c), g + r * ldg + c, 16);
  }
}
// the same for a whole tile of zero-padded rows, by plain stores
__device__ __forceinline__ void zero_rows(bf16 *s, int lds, int r0, int r1, int nt)
{
  for (int e = threadIdx.x; e < (r1 - r0) * lds; e += nt) s[r0 * lds + e] = __float2bfloat16(0.f);
}

// fragments: A stored m-major (k contiguous) or k-major; B stored k-major (n contiguous) or n-major
__device__ __forceinline__ void frag_a(uint32_t *f, const bf16 *s, int lds, int m0, int k0)
{
  const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
  ldsm_x4(f, smem_addr(s + (m0 + (mat & 1) * 8 + r) * lds + k0 + (mat >> 1) * 8), false);
}
__device__ __forceinline__ void frag_at(uint32_t *f, const bf16 *s, int lds, int m0, int k0)
{
  const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
  ldsm_x4(f, smem_addr(s + (k0 + (mat >> 1) * 8 + r) * lds + m0 + (mat & 1) * 8), true);
}
// two n tiles of 8: f[0..1] columns n0 .. n0 + 7, f[2..3] columns n0 + 8 .. n0 + 15
__device__ __forceinline__ void frag_b(uint32_t *f, const bf16 *s, int lds, int n0, int k0)
{
  const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
  ldsm_x4(f, smem_addr(s + (k0 + (mat & 1) * 8 + r) * lds + n0 + (mat >> 1) * 8), true);
}
__device__ __forceinline__ void frag_bt(uint32_t *f, const bf16 *s, int lds, int n0, int k0)
{
  const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
  ldsm_x4(f, smem_addr(s + (n0 + (mat >> 1) * 8 + r) * lds + k0 + (mat & 1) * 8), false);
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ uint32_t pack_bf16(float x, float y)
{
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u)
{
  const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162 *>(&u);
  return make_float2(__low2float(v), __high2float(v));
}

// GELU of two values, rounded to BF16: the bits of pack_bf16(gelu_f(x), gelu_f(y)) for some 20 instead of
// 50 instructions a value.  erfc from the rational formula 7.1.26 of Abramowitz and Stegun (Hastings;
// within 1.5e-7), which gives GELU within GELU_ERR |x| of gelu_f's value; where both ends of
// that interval round to the same BF16 numbers these are the result, else (four values in a
// thousand) gelu_f decides.  tests/test_nn_gelu.py compares every float (the largest difference from
// gelu_f measured is 3.9e-7 |x|).  A forward row kernel at 64 samples 133 -> 122 us, 64 draws served
// in 593 -> 567 us.
constexpr float GELU_ERR = 5e-7f;
__device__ __forceinline__ float gelu_near(float x)
{
  float t, e;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(fabsf(x), 0.3275911f * 0.70710678f, 1.0f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * x * -0.72134752f));   // exp(-x^2 / 2)
  float q = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
  q = fmaf(q, t, 0.5f * 1.421413741f);
  q = fmaf(q, t, 0.5f * -0.284496736f);
  q = fmaf(q, t, 0.5f * 0.254829592f) * t * e;                                // erfc(|x| / sqrt 2) / 2
  return x * (x >= 0.0f ? 1.0f - q : q);
}
__device__ __forceinline__ uint32_t gelu_pack(float x, float y)
{
  const float gx = gelu_near(x), gy = gelu_near(y);
  const uint32_t lo = pack_bf16(fmaf(x, -GELU_ERR, gx), fmaf(y, -GELU_ERR, gy));
  const uint32_t hi = pack_bf16(fmaf(x, GELU_ERR, gx), fmaf(y, GELU_ERR, gy));
  return lo == hi ? lo : pack_bf16(gelu_f(x), gelu_f(y));
}

// GELU' of a BF16 pre-activation from a table in shared memory: the values of gelu_grad_f at the
// BF16 numbers of magnitude 2^-8 to 4 (10 binades, both signs: 10 KB), the function itself
// outside.  The function costs some 45 instructions, the look-up 6 and one conflicted read.
constexpr int GLUT_LO = (127 - 8) << 7, GLUT_N = 10 << 7, GLUT = 2 * GLUT_N;
__device__ __forceinline__ float gelu_grad_lut(uint32_t bits, const float *lut)
{
  const uint32_t i = (bits & 0x7fffu) - GLUT_LO;
  if (i < GLUT_N) return lut[i + ((bits & 0x8000u) ? GLUT_N : 0)];
  return gelu_grad_f(__uint_as_float(bits << 16));
}
__device__ __forceinline__ void load_gelu_lut(float *s, const float *lut, int nt)
{
  for (int e = threadIdx.x; e < GLUT / 4; e += nt) reinterpret_cast<float4 *>(s)[e] = reinterpret_cast<const float4 *>(lut)[e];
}
__global__ void gelu_lut_kernel(float *lut)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < GLUT) {
    const uint32_t bits = (uint32_t)(GLUT_LO + i % GLUT_N) | (i < GLUT_N ? 0u : 0x8000u);
    lut[i] = gelu_grad_f(__uint_as_float(bits << 16));
  }
}

enum { ROW_LIFT = 0, ROW_FWD = 1, ROW_BWD = 2, ROW_TOP = 3 };

struct RowArgs {
  const bf16 *in;        // [rows][nx][W]: FWD H, BWD dA of the layer above (LIFT [rows][nx][cin])
  const bf16 *spec;      // [rows][m2][W]: FWD the layer's spectrum after the inverse y transform, BWD its adjoint
  const bf16 *wt;        // FWD, LIFT [K][W]; BWD [W][W], applied transposed
  const float *bias;     // FWD, LIFT
  const bf16 *einv;      // [nx][m2]: spectrum row -> pixels
  const bf16 *efwd;      // [m2][nx]: pixels -> spectrum row
  const bf16 *pre;       // BWD: pre-activation of the layer below (null: none)
  const float *lut;      // BWD: GELU' table
  bf16 *out;             // [rows][nx][W]: H, or dA (dH below the first layer)
  bf16 *aux;             // FWD: pre-activation (null: not stored)
  bf16 *spec_out;        // [rows][m2][W] (null: none)
  int rows, nx, m2, cin;
  // TOP: the decoder's data gradient [B][nrec][ny][W], summed into the receivers' columns
  const bf16 *dd0;
  const int *rec_x;
  int nrec, ny;
};

template <int W, int KIND>
struct RowSmem {
  static constexpr int LW = W + 8;
  static constexpr int KIN = (KIND == ROW_LIFT) ? 64 : W;   // widest convolution input
  static __host__ __device__ size_t wt() { return (KIND == ROW_TOP) ? 0 : (size_t)KIN * LW; }
  static __host__ __device__ size_t efwd(int nx) { return (size_t)RK * (nx + 8); }
  static __host__ __device__ size_t in(int nx, int cin) { return (size_t)nx * ((KIND == ROW_LIFT) ? cin + 8 : LW); }
  static __host__ __device__ size_t spec() { return (KIND == ROW_FWD || KIND == ROW_BWD) ? (size_t)RK * LW : 0; }
  static __host__ __device__ size_t stage(int nx, int cin) { return in(nx, cin) + spec(); }
  static __host__ __device__ size_t out(int nx) { return (KIND == ROW_LIFT) ? (size_t)nx * LW : 0; }
  static __host__ __device__ size_t bytes(int nx, int cin)
  {
    return 2 * (wt() + efwd(nx) + (KIND == ROW_TOP ? 1 : 2) * stage(nx, cin) + out(nx)) + (W + (KIND == ROW_BWD ? GLUT : 0)) * sizeof(float);
  }
};

// rows [m0, m0 + 16), channels [c0, c0 + CW) of a shared tile -> global memory, 16 bytes a lane, by
// one warp
template <int W, int CW>
__device__ __forceinline__ void store_rows16(bf16 *g, const bf16 *s, int m0, int c0)
{
  constexpr int PER = CW / 8;
  for (int e = threadIdx.x & 31; e < 16 * PER; e += 32) {
    const int r = e / PER, c = c0 + (e - r * PER) * 8;
    *reinterpret_cast<uint4 *>(g + (size_t)(m0 + r) * W + c) = *reinterpret_cast<const uint4 *>(s + (m0 + r) * (W + 8) + c);
  }
}

// spectrum row [m2][W] of a row of pixels in shared memory: efwd (RK x nx, zero rows past m2)
template <int W>
__device__ __forceinline__ void x_analysis(const bf16 *sE, const bf16 *px, int nx, int m2, bf16 *out)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int mt = warp & 1, np = warp >> 1;   // 16 spectrum rows x 16 channels per warp
  if (np * 16 >= W || mt * 16 >= m2) return;
  float acc[2][4] = {};
  for (int k = 0; k < nx; k += 16) {
    uint32_t a[4], b[4];
    frag_a(a, sE, nx + 8, mt * 16, k);
    frag_b(b, px, W + 8, np * 16, k);
    mma_bf16(acc[0], a, b);
    mma_bf16(acc[1], a, b + 2);
  }
#pragma unroll
  for (int t = 0; t < 2; t++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = mt * 16 + gid + 8 * h;
      if (r < m2) *reinterpret_cast<uint32_t *>(out + (size_t)r * W + np * 16 + t * 8 + tig * 2) = pack_bf16(acc[t][2 * h], acc[t][2 * h + 1]);
    }
}

// Persistent over the image rows, two stages of asynchronous copies.  A warp owns 16 pixels
// through the convolution and activation: it holds them in operand registers, so results (and, on
// their way, the pre-activations) replace them in shared memory without a block barrier; the
// x transform at the end reads all pixels.  What bounds it is issue and the latency of dependent
// instructions (40 instructions per value, half of them the activation, 61 % of the issue slots) at the
// warps that fit: 32 channels at a time and no second stage for the pre-activations leave three
// CTAs per SM (80 registers, 74 KB).
template <int W, int KIND>
__global__ void __launch_bounds__(RT, 3) row_kernel(const RowArgs a)
{
  typedef RowSmem<W, KIND> L;
  constexpr int LW = L::LW, NT = W / 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  bf16 *sW = reinterpret_cast<bf16 *>(rsm);
  bf16 *sE = sW + L::wt();
  bf16 *st0 = sE + L::efwd(a.nx);
  bf16 *sO = st0 + (KIND == ROW_TOP ? 1 : 2) * L::stage(a.nx, a.cin);
  float *sB = reinterpret_cast<float *>(sO + L::out(a.nx)), *sG = sB + W;
  const int nx = a.nx, m2 = a.m2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  __shared__ int rec[KIND == ROW_TOP ? RNX : 1], more[KIND == ROW_TOP ? RREC : 1];   // TOP: a column's first receiver, the next of a receiver
  const int kin = (KIND == ROW_LIFT) ? a.cin : W, lin = (KIND == ROW_LIFT) ? a.cin + 8 : LW;
  constexpr bool SPEC = KIND == ROW_FWD || KIND == ROW_BWD;

  // tables, zero-padded to whole k steps
  if (KIND != ROW_TOP) copy_tile<W>(sW, LW, a.wt, W, kin, W, RT);
  for (int e = threadIdx.x; e < RK * (nx + 8); e += RT) {
    const int r = e / (nx + 8), c = e - r * (nx + 8);
    sE[e] = (r < m2 && c < nx) ? a.efwd[r * nx + c] : __float2bfloat16(0.f);
  }
  // a warp's pixels are the same columns of every row: its part of the inverse x transform stays in
  // operand registers (row gid + 8 (i % 2), k pair 2 tig + 8 (i / 2) of a k step)
  uint32_t fe[RK / 16][4];
  if (SPEC) {
#pragma unroll
    for (int k = 0; k < RK / 16; k++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = warp * 16 + gid + 8 * (i & 1), c = k * 16 + tig * 2 + 8 * (i >> 1);
        fe[k][i] = (r < nx && c < m2) ? *reinterpret_cast<const uint32_t *>(a.einv + r * m2 + c) : 0u;
      }
    for (int s = 0; s < 2; s++) zero_rows(st0 + s * L::stage(nx, a.cin) + L::in(nx, a.cin), LW, m2, RK, RT);
  }
  if (KIND == ROW_BWD && a.pre) load_gelu_lut(sG, a.lut, RT);
  if (KIND == ROW_LIFT || KIND == ROW_FWD)
    for (int e = threadIdx.x; e < W; e += RT) sB[e] = a.bias[e];
  if (KIND == ROW_TOP)
    for (int x = threadIdx.x; x < nx; x += RT) {   // (one thread per column: its receivers in ascending order)
      int first = -1, last = -1;
      for (int r = 0; r < a.nrec; r++)
        if (a.rec_x[r] == x) {
          if (first < 0) first = r;
          else more[last] = r;
          last = r;
          more[r] = -1;
        }
      rec[x] = first;
    }

  auto load = [&](int row, int s) {
    bf16 *st = st0 + s * L::stage(nx, a.cin);
    if (KIND != ROW_LIFT) copy_tile<W>(st, lin, a.in + (size_t)row * nx * kin, kin, nx, kin, RT);
    else if (kin == 16) copy_tile<16>(st, lin, a.in + (size_t)row * nx * kin, kin, nx, kin, RT);
    else copy_tile(st, lin, a.in + (size_t)row * nx * kin, kin, nx, kin, RT);
    if (SPEC) copy_tile<W>(st + L::in(nx, a.cin), LW, a.spec + (size_t)row * m2 * W, W, m2, W, RT);
      };
  if (KIND != ROW_TOP) {
    if ((int)blockIdx.x < a.rows) load(blockIdx.x, 0);
    cp_async_commit();
  }
  int s = 0;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x, s ^= 1) {
    bf16 *px = st0;   // the row's pixels [nx][LW], input and then result
    if (KIND == ROW_TOP) {
      const int b = row / a.ny, y = row - b * a.ny;
      __syncthreads();   // (the previous row's x transform has read px)
      for (int e = threadIdx.x; e < nx * NT; e += RT) {
        const int x = e / NT, c = (e - x * NT) * 8;
        float v[8] = {};
        for (int r = rec[x]; r >= 0; r = more[r]) {
          const uint4 q = *reinterpret_cast<const uint4 *>(a.dd0 + (((size_t)b * a.nrec + r) * a.ny + y) * W + c);
          const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float2 f = unpack_bf16(u[i]);
            v[2 * i] += f.x;
            v[2 * i + 1] += f.y;
          }
        }
        const uint4 o = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
        *reinterpret_cast<uint4 *>(px + x * LW + c) = o;
        *reinterpret_cast<uint4 *>(a.out + ((size_t)row * nx + x) * W + c) = o;
      }
    } else {
      bf16 *st = st0 + s * L::stage(nx, a.cin);
      cp_async_wait<0>();
      __syncthreads();
      px = (KIND == ROW_LIFT) ? sO : st;
      const int m0 = warp * 16;
      const bool on = m0 < nx, pre = KIND == ROW_BWD && a.pre;
      uint32_t fp[L::KIN / 16][4];
      if (on) {
#pragma unroll
        for (int k = 0; k < L::KIN / 16; k++)
          if (k * 16 < kin) frag_a(fp[k], st, lin, m0, k * 16);
        __syncwarp();   // the warp's pixels have been read
        if (pre)        // the pre-activations take their place
          for (int e = lane; e < 16 * NT; e += 32)
            cp_async16(smem_addr(px + (m0 + e / NT) * LW + (e % NT) * 8), a.pre + ((size_t)row * nx + m0 + e / NT) * W + (e % NT) * 8, 16);
      }
      cp_async_commit();
      if (row + (int)gridDim.x < a.rows) load(row + gridDim.x, s ^ 1);   // (freed by the barrier that ended the previous row)
      cp_async_commit();
      if (on) {
        const bf16 *sS = st + L::in(nx, a.cin);
        constexpr int CW = (W % 32 == 0) ? 32 : 16, CT = CW / 8;   // channels at a time
#pragma unroll
        for (int c0 = 0; c0 < W; c0 += CW) {
          // spectrum row -> pixels, and the 1x1 convolution
          float sp[CT][4] = {}, cv[CT][4] = {};
          uint32_t fb[4];
          if (SPEC)
#pragma unroll
            for (int k = 0; k < RK / 16; k++)
#pragma unroll
              for (int n = 0; n < CT; n += 2) {
                frag_b(fb, sS, LW, c0 + n * 8, k * 16);
                mma_bf16(sp[n], fe[k], fb);
                mma_bf16(sp[n + 1], fe[k], fb + 2);
              }
#pragma unroll
          for (int k = 0; k < L::KIN / 16; k++)
            if (k * 16 < kin)
#pragma unroll
              for (int n = 0; n < CT; n += 2) {
                if (KIND == ROW_BWD) frag_bt(fb, sW, LW, c0 + n * 8, k * 16);
                else frag_b(fb, sW, LW, c0 + n * 8, k * 16);
                mma_bf16(cv[n], fp[k], fb);
                mma_bf16(cv[n + 1], fp[k], fb + 2);
              }
          if (pre && c0 == 0) {
            cp_async_wait<1>();
            __syncwarp();
          }
          if (KIND == ROW_FWD) {
            // the pre-activation, through px to memory where it is kept
#pragma unroll
            for (int n = 0; n < CT; n++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int c = c0 + n * 8 + tig * 2;
                cv[n][2 * h] = cv[n][2 * h] + round_bf16(sp[n][2 * h]) + sB[c];
                cv[n][2 * h + 1] = cv[n][2 * h + 1] + round_bf16(sp[n][2 * h + 1]) + sB[c + 1];
                if (a.aux) *reinterpret_cast<uint32_t *>(px + (m0 + gid + 8 * h) * LW + c) = pack_bf16(cv[n][2 * h], cv[n][2 * h + 1]);
              }
            if (a.aux) {
              __syncwarp();
              store_rows16<W, CW>(a.aux + (size_t)row * nx * W, px, m0, c0);
              __syncwarp();
            }
          }
#pragma unroll
          for (int n = 0; n < CT; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int c = c0 + n * 8 + tig * 2;
              uint32_t *at = reinterpret_cast<uint32_t *>(px + (m0 + gid + 8 * h) * LW + c);
              float x = cv[n][2 * h], y = cv[n][2 * h + 1];
              if (KIND == ROW_LIFT) {
                x += sB[c];
                y += sB[c + 1];
              } else if (KIND != ROW_FWD) {
                x = sp[n][2 * h] + round_bf16(x);
                y = sp[n][2 * h + 1] + round_bf16(y);
                if (pre) {
                  const uint32_t q = *at;
                  x = round_bf16(x) * gelu_grad_lut(q & 0xffffu, sG);
                  y = round_bf16(y) * gelu_grad_lut(q >> 16, sG);
                }
              }
              *at = (KIND == ROW_FWD) ? gelu_pack(x, y) : pack_bf16(x, y);
            }
        }
        __syncwarp();
        store_rows16<W, W>(a.out + (size_t)row * nx * W, px, m0, 0);
      }
    }
    if (a.spec_out) {
      __syncthreads();
      x_analysis<W>(sE, px, nx, m2, a.spec_out + (size_t)row * m2 * W);
    }
    if (KIND != ROW_TOP) __syncthreads();   // this stage is free for the row after the next
  }
}

// The last layer at the receivers' pixels only (the decoder reads nothing else): one warp per
// image row, 16 receivers at a time, D0[b][r][y][W] = bf16(conv + spectral + bias).
struct LastArgs {
  const bf16 *in, *spec, *wt, *einv;
  const float *bias;
  const int *rec_x;
  bf16 *d0;
  int rows, nx, ny, m2, nrec;
};
template <int W>
constexpr size_t last_smem() { return 2 * ((size_t)W * (W + 8) + 8 * ((size_t)RK * (W + 8) + 16 * (W + 8) + 16 * (RK + 8))); }

template <int W>
__global__ void __launch_bounds__(RT) last_kernel(const LastArgs a)
{
  constexpr int LW = W + 8, LE = RK + 8, NT = W / 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  bf16 *sW = reinterpret_cast<bf16 *>(rsm);
  bf16 *sS = sW + W * LW + warp * (RK * LW + 16 * LW + 16 * LE), *sH = sS + RK * LW, *sI = sH + 16 * LW;
  copy_tile<W>(sW, LW, a.wt, W, W, W, RT);
  cp_async_commit();
  const int row = blockIdx.x * 8 + warp;
  const bool on = row < a.rows;
  const int b = row / a.ny, y = row - b * a.ny;
  if (on) {
    for (int e = lane; e < a.m2 * NT; e += 32)
      cp_async16(smem_addr(sS + (e / NT) * LW + (e % NT) * 8), a.spec + ((size_t)row * a.m2 + e / NT) * W + (e % NT) * 8, 16);
    for (int e = lane; e < (RK - a.m2) * LW; e += 32) sS[a.m2 * LW + e] = __float2bfloat16(0.f);
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncthreads();
  if (!on) return;
  for (int r0 = 0; r0 < a.nrec; r0 += 16) {
    __syncwarp();
    for (int e = lane; e < 16 * NT; e += 32) {
      const int r = e / NT, x = (r0 + r < a.nrec) ? a.rec_x[r0 + r] : 0;
      cp_async16(smem_addr(sH + r * LW + (e % NT) * 8), a.in + ((size_t)row * a.nx + x) * W + (e % NT) * 8, 16);
    }
    cp_async_commit();
    for (int e = lane; e < 16 * LE; e += 32) {
      const int r = e / LE, c = e - r * LE, x = (r0 + r < a.nrec) ? a.rec_x[r0 + r] : 0;
      sI[e] = (c < a.m2) ? a.einv[x * a.m2 + c] : __float2bfloat16(0.f);
    }
    cp_async_wait<0>();
    __syncwarp();
    float sp[NT][4] = {}, cv[NT][4] = {};
#pragma unroll
    for (int k = 0; k < RK; k += 16) {
      uint32_t fa[4], fb[4];
      frag_a(fa, sI, LE, 0, k);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        frag_b(fb, sS, LW, n * 8, k);
        mma_bf16(sp[n], fa, fb);
        mma_bf16(sp[n + 1], fa, fb + 2);
      }
    }
#pragma unroll
    for (int k = 0; k < W; k += 16) {
      uint32_t fa[4], fb[4];
      frag_a(fa, sH, LW, 0, k);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        frag_b(fb, sW, LW, n * 8, k);
        mma_bf16(cv[n], fa, fb);
        mma_bf16(cv[n + 1], fa, fb + 2);
      }
    }
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = n * 8 + tig * 2, r = r0 + gid + 8 * h;
        if (r < a.nrec)
          *reinterpret_cast<uint32_t *>(a.d0 + (((size_t)b * a.nrec + r) * a.ny + y) * W + c) =
              pack_bf16(cv[n][2 * h] + round_bf16(sp[n][2 * h]) + a.bias[c], cv[n][2 * h + 1] + round_bf16(sp[n][2 * h + 1]) + a.bias[c + 1]);
      }
  }
}

// ---- y transforms: A [4m][2ny] (k contiguous) shared by the samples; 128 columns (kx, c) per
// CTA, so that a batch of 32 is one wave at two CTAs per SM (batch 32, analysis and
// synthesis: 64 columns, 512 CTAs of 70 KB in 456 places, 18 and 15 us; 128 columns 10 and 10)
constexpr int YN = 128, YL = YN + 8;
struct YArgs {
  const bf16 *A;         // My [4m][2ny], or its transpose [2ny][4m] for the synthesis
  const bf16 *B;         // analysis [b][2ny][m w]; synthesis [b][4m][m w]
  bf16 *C;               // analysis: mode-major [(j, kx)][b][part][w]; synthesis [b][2ny][m w]
  int ny, m, batch;
};
__host__ __device__ inline size_t y_analysis_smem(int ny) { return 2 * ((size_t)64 * (2 * ny + 8) + (size_t)2 * ny * YL); }
__host__ __device__ inline size_t y_synthesis_smem(int ny) { return 2 * ((size_t)2 * ny * 72 + (size_t)64 * YL + (size_t)8 * 16 * YL); }

// copies of the YN columns from n0 of rows k0 .. k1 (zero past column N)
__device__ __forceinline__ void copy_cols(bf16 *s, const bf16 *g, long ldg, int k0, int k1, int n0, int N)
{
  for (int e = threadIdx.x; e < (k1 - k0) * (YN / 8); e += RT) {
    const int r = k0 + e / (YN / 8), c = (e % (YN / 8)) * 8;
    const bool in = n0 + c < N;   // (N is a multiple of 16)
    cp_async16(smem_addr(s + r * YL + c), in ? g + r * ldg + n0 + c : g, in ? 16 : 0);
  }
}

// warp w: rows 16 (w % 4) .., columns 64 (w / 4) ..
template <int W>
__global__ void __launch_bounds__(RT, 2) y_analysis(const YArgs a)
{
  extern __shared__ __align__(16) unsigned char rsm[];
  const int K = 2 * a.ny, LA = K + 8, M = 4 * a.m, N = a.m * W, n0 = blockIdx.x * YN, b = blockIdx.y;
  bf16 *sA = reinterpret_cast<bf16 *>(rsm), *sB = sA + 64 * LA;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int m0 = (warp & 3) * 16, c0 = (warp >> 2) * 64;
  // everything in flight at once, in four parts of k that are computed as they land
  constexpr int part = 2 * RNY / 4;
  for (int q = 0; q < 4; q++) {
    const int k0 = min(q * part, K), k1 = min(k0 + part, K);
    for (int e = threadIdx.x; e < M * (part / 8); e += RT) {
      const int r = e / (part / 8), c = k0 + (e % (part / 8)) * 8;
      if (c < k1) cp_async16(smem_addr(sA + r * LA + c), a.A + (size_t)r * K + c, 16);
    }
    copy_cols(sB, a.B + (size_t)b * K * N, N, k0, k1, n0, N);
    cp_async_commit();
  }
  zero_rows(sA, LA, M, 64, RT);
  float acc[8][4] = {};
  for (int q = 0; q < 4; q++) {
    if (q == 0) cp_async_wait<3>();
    else if (q == 1) cp_async_wait<2>();
    else if (q == 2) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    if (m0 >= M) continue;
    for (int k = min(q * part, K); k < min((q + 1) * part, K); k += 16) {
      uint32_t fa[4], fb[4];
      frag_a(fa, sA, LA, m0, k);
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        frag_b(fb, sB, YL, c0 + n * 8, k);
        mma_bf16(acc[n], fa, fb);
        mma_bf16(acc[n + 1], fa, fb + 2);
      }
    }
  }
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = m0 + gid + 8 * h, col = n0 + c0 + n * 8 + tig * 2;
      if (r >= M || col >= N) continue;
      const int j = r >> 1, pt = r & 1, kx = col / W, c = col - kx * W;
      *reinterpret_cast<uint32_t *>(a.C + (((size_t)(j * a.m + kx) * a.batch + b) * 2 + pt) * W + c) = pack_bf16(acc[n][2 * h], acc[n][2 * h + 1]);
    }
}

// warp w: rows 16 w, 16 w + 128, ..; its 16 x YN results leave through a patch of shared memory in
// 16-byte stores
template <int W>
__global__ void __launch_bounds__(RT, 2) y_synthesis(const YArgs a)
{
  extern __shared__ __align__(16) unsigned char rsm[];
  const int K = 4 * a.m, K16 = (K + 15) / 16 * 16, M = 2 * a.ny, N = a.m * W, n0 = blockIdx.x * YN, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  bf16 *sA = reinterpret_cast<bf16 *>(rsm), *sB = sA + M * 72, *sO = sB + 64 * YL + warp * 16 * YL;
  copy_cols(sB, a.B + (size_t)b * K * N, N, 0, K, n0, N);
  zero_rows(sB, YL, K, K16, RT);
  if (K % 8 == 0) {
    for (int e = threadIdx.x; e < M * 8; e += RT)
      if ((e & 7) * 8 < K) cp_async16(smem_addr(sA + (e >> 3) * 72 + (e & 7) * 8), a.A + (size_t)(e >> 3) * K + (e & 7) * 8, 16);
    if (K16 > K)
      for (int e = threadIdx.x; e < M * (K16 - K); e += RT) sA[(e / (K16 - K)) * 72 + K + e % (K16 - K)] = __float2bfloat16(0.f);
  } else {
    for (int e = threadIdx.x; e < M * K16; e += RT) {
      const int r = e / K16, c = e - r * K16;
      sA[r * 72 + c] = (c < K) ? a.A[(size_t)r * K + c] : __float2bfloat16(0.f);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  for (int m0 = warp * 16; m0 < M; m0 += 128) {
#pragma unroll
    for (int half = 0; half < 2; half++) {
      float acc[8][4] = {};
      for (int k = 0; k < K16; k += 16) {
        uint32_t fa[4], fb[4];
        frag_a(fa, sA, 72, m0, k);
#pragma unroll
        for (int n = 0; n < 8; n += 2) {
          frag_b(fb, sB, YL, half * 64 + n * 8, k);
          mma_bf16(acc[n], fa, fb);
          mma_bf16(acc[n + 1], fa, fb + 2);
        }
      }
#pragma unroll
      for (int n = 0; n < 8; n++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          *reinterpret_cast<uint32_t *>(sO + (gid + 8 * h) * YL + half * 64 + n * 8 + tig * 2) = pack_bf16(acc[n][2 * h], acc[n][2 * h + 1]);
    }
    __syncwarp();
    for (int e = lane; e < 16 * (YN / 8); e += 32) {
      const int r = e / (YN / 8), c = (e % (YN / 8)) * 8;
      if (n0 + c < N) *reinterpret_cast<uint4 *>(a.C + ((size_t)b * M + m0 + r) * N + n0 + c) = *reinterpret_cast<const uint4 *>(sO + r * YL + c);
    }
    __syncwarp();
  }
}

// ---- channel mixing of one mode: [Zre Zim] [[Wre Wim] [-Wim Wre]] per sample, k ascending over
// (part, channel).  The block matrix is never formed: -Wim is Wim with its sign bits flipped.
struct ModeArgs {
  const bf16 *Z;           // [mode][b][2][w]
  const bf16 *Wre, *Wim;   // [mode][w][w]
  bf16 *Y;                 // [b][j][part][kx][w]
  const bf16 *dY;          // mode_grad: [mode][b][2][w]
  float *dWre, *dWim;      // mode_grad: [mode][w][w]
  int m, batch;
};
constexpr int MB = 32;   // samples per pass
template <int W> constexpr size_t mode_smem() { return 2 * ((size_t)2 * W * (W + 8) + (size_t)MB * (2 * W + 8)); }

template <int W>
__device__ __forceinline__ void mode_load_z(bf16 *s, const bf16 *g, int rows)
{
  constexpr int LZ = 2 * W + 8;
  copy_tile<2 * W>(s, LZ, g, 2 * W, rows, 2 * W, RT);
  zero_rows(s, LZ, rows, MB, RT);
}

// TRANS: the adjoint (dZ = dY Wblk^T)
template <int W, bool TRANS>
__device__ __forceinline__ void mode_product(const bf16 *sZ, const bf16 *sRe, const bf16 *sIm, bf16 *Y, int mode, int m, int b0, int batch)
{
  constexpr int LW = W + 8, LZ = 2 * W + 8, NP = 2 * W / 16;   // column pairs of tiles
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int j = mode / m, kx = mode - j * m;
  for (int u = warp; u < NP * (MB / 16); u += RT / 32) {
    const int mt = u & 1, n0 = (u >> 1) * 16, po = n0 / W, co = n0 - po * W;
    if (b0 + mt * 16 >= batch) continue;
    float acc[2][4] = {};
#pragma unroll
    for (int pi = 0; pi < 2; pi++) {
      // block (pi, po) of the mixing matrix, or (po, pi) of its transpose
      const bf16 *w = (pi == po) ? sRe : sIm;
      const uint32_t flip = (pi != po && (TRANS ? po == 1 : pi == 1)) ? 0x80008000u : 0u;
#pragma unroll
      for (int k = 0; k < W; k += 16) {
        uint32_t fa[4], fb[4];
        frag_a(fa, sZ, LZ, mt * 16, pi * W + k);
        if (TRANS) frag_bt(fb, w, LW, co, k);
        else frag_b(fb, w, LW, co, k);
#pragma unroll
        for (int i = 0; i < 4; i++) fb[i] ^= flip;
        mma_bf16(acc[0], fa, fb);
        mma_bf16(acc[1], fa, fb + 2);
      }
    }
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int b = b0 + mt * 16 + gid + 8 * h;
        if (b < batch)
          *reinterpret_cast<uint32_t *>(Y + ((((size_t)b * 2 * m + j) * 2 + po) * m + kx) * W + co + t * 8 + tig * 2) =
              pack_bf16(acc[t][2 * h], acc[t][2 * h + 1]);
      }
  }
}

template <int W>
__global__ void __launch_bounds__(RT) mode_mix(const ModeArgs a)
{
  constexpr int LW = W + 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  bf16 *sRe = reinterpret_cast<bf16 *>(rsm), *sIm = sRe + W * LW, *sZ = sIm + W * LW;
  const int mode = blockIdx.x;
  copy_tile<W>(sRe, LW, a.Wre + (size_t)mode * W * W, W, W, W, RT);
  copy_tile<W>(sIm, LW, a.Wim + (size_t)mode * W * W, W, W, W, RT);
  for (int b0 = 0; b0 < a.batch; b0 += MB) {
    if (b0) __syncthreads();
    mode_load_z<W>(sZ, a.Z + ((size_t)mode * a.batch + b0) * 2 * W, min(MB, a.batch - b0));
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    mode_product<W, false>(sZ, sRe, sIm, a.Y, mode, a.m, b0, a.batch);
  }
}

// The adjoint of the mixing (dZ, stored like Y) and the gradients of Wre and Wim of one mode:
// with d = [Zre Zim]^T [dYre dYim], k over the samples, dWre = d(re,re) + d(im,im) and
// dWim = d(re,im) - d(im,re).
template <int W> constexpr size_t mode_grad_smem() { return 2 * ((size_t)2 * W * (W + 8) + (size_t)2 * MB * (2 * W + 8)); }

template <int W>
__global__ void __launch_bounds__(RT) mode_grad(const ModeArgs a)
{
  constexpr int LW = W + 8, LZ = 2 * W + 8, T = W / 16, U = (T * T + 7) / 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  bf16 *sRe = reinterpret_cast<bf16 *>(rsm), *sIm = sRe + W * LW, *sZ = sIm + W * LW, *sY = sZ + MB * LZ;
  const int mode = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  copy_tile<W>(sRe, LW, a.Wre + (size_t)mode * W * W, W, W, W, RT);
  copy_tile<W>(sIm, LW, a.Wim + (size_t)mode * W * W, W, W, W, RT);
  float acc[U][4][2][4] = {};   // re-re, im-im, re-im, im-re
  for (int b0 = 0; b0 < a.batch; b0 += MB) {
    if (b0) __syncthreads();
    const int rows = min(MB, a.batch - b0);
    mode_load_z<W>(sZ, a.Z + ((size_t)mode * a.batch + b0) * 2 * W, rows);
    mode_load_z<W>(sY, a.dY + ((size_t)mode * a.batch + b0) * 2 * W, rows);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    mode_product<W, true>(sY, sRe, sIm, a.Y, mode, a.m, b0, a.batch);
    for (int k = 0; k < rows; k += 16)
#pragma unroll
      for (int i = 0; i < U; i++) {
        const int u = warp + 8 * i, ci = (u / T) * 16, co = (u % T) * 16;
        if (u >= T * T) break;
        uint32_t zr[4], zi[4], yr[4], yi[4];
        frag_at(zr, sZ, LZ, ci, k);
        frag_at(zi, sZ, LZ, W + ci, k);
        frag_b(yr, sY, LZ, co, k);
        frag_b(yi, sY, LZ, W + co, k);
#pragma unroll
        for (int t = 0; t < 2; t++) {
          mma_bf16(acc[i][0][t], zr, yr + 2 * t);
          mma_bf16(acc[i][1][t], zi, yi + 2 * t);
          mma_bf16(acc[i][2][t], zr, yi + 2 * t);
          mma_bf16(acc[i][3][t], zi, yr + 2 * t);
        }
      }
  }
#pragma unroll
  for (int i = 0; i < U; i++) {
    const int u = warp + 8 * i, ci = (u / T) * 16, co = (u % T) * 16;
    if (u >= T * T) break;
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const size_t o = ((size_t)mode * W + ci + gid + 8 * h) * W + co + t * 8 + tig * 2;
        *reinterpret_cast<float2 *>(a.dWre + o) =
            make_float2(acc[i][0][t][2 * h] + acc[i][1][t][2 * h], acc[i][0][t][2 * h + 1] + acc[i][1][t][2 * h + 1]);
        *reinterpret_cast<float2 *>(a.dWim + o) =
            make_float2(acc[i][2][t][2 * h] - acc[i][3][t][2 * h], acc[i][2][t][2 * h + 1] - acc[i][3][t][2 * h + 1]);
      }
  }
}

// ---- weight gradient of a 1x1 convolution: partial[chunk] (R x W) = X^T dY over kc pixels, k
// ascending; X [pixels][R], dY [pixels][W].  Where kc is a multiple of CSP, also the column sums of
// dY over every CSP pixels (sums: [pixels / CSP][W]) while its rows are in shared memory: RT / W
// lanes per column, each over every (RT / W)-th pixel, added in lane order.
// At batch 32 there are 256 chunks for 152 SMs: two stages of copies ahead of the one in use keep
// enough bytes in flight (one ahead: 41 us; half the columns per CTA: 57).
constexpr int WGK = 128, WGS = 3, CSP = 1024;   // pixels per stage, stages, pixels per column sum
template <int W> size_t wgrad_smem(int R) { return 2 * (size_t)WGS * WGK * (R + 8 + W + 8); }

// (RC: R where it is known, else 0; WHOLE: kc is a multiple of WGK -- both let the inner loop unroll
// with fixed addresses)
template <int W, int RC, bool WHOLE>
__global__ void __launch_bounds__(RT) weight_grad_partial(const bf16 *X, int r_dyn, const bf16 *dY, int kc, float *partial, float *sums)
{
  constexpr int LW = W + 8, NP = W / 16, U = RC ? (RC / 16 * NP + 7) / 8 : 2;   // 16 x 16 tiles, at most 4 x 4 over 8 warps
  const int R = RC ? RC : r_dyn;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int LR = R + 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const size_t p0 = (size_t)blockIdx.x * kc;
  bf16 *st = reinterpret_cast<bf16 *>(rsm);
  const int stage = WGK * (LR + LW), nst = (kc + WGK - 1) / WGK, units = (R / 16) * NP;
  auto load = [&](int i) {
    if (i < nst) {
      bf16 *s = st + (i % WGS) * stage;
      const int n = min(WGK, kc - i * WGK);
      copy_tile<RC>(s, LR, X + (p0 + (size_t)i * WGK) * R, R, n, R, RT);
      copy_tile<W>(s + WGK * LR, LW, dY + (p0 + (size_t)i * WGK) * W, W, n, W, RT);
    }
    cp_async_commit();
  };
  constexpr int LANES = RT / W, W2 = W / 2;
  __shared__ float sc[RT];
  const int lane_c = threadIdx.x / W2, col = (threadIdx.x % W2) * 2;   // two columns a thread
  int next = lane_c;   // this lane's next pixel of the column sum
  float csum0 = 0.f, csum1 = 0.f;
  for (int i = 0; i < WGS - 1; i++) load(i);
  float acc[U][2][4] = {};
  for (int i = 0; i < nst; i++) {
    load(i + WGS - 1);   // (its stage was freed by the barrier that ended the previous pass)
    cp_async_wait<WGS - 1>();
    __syncthreads();
    const bf16 *sX = st + (i % WGS) * stage, *sY = sX + WGK * LR;
    const int kn = WHOLE ? WGK : min(WGK, kc - i * WGK);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = warp + 8 * u;
      if (t < units) {
#pragma unroll(WHOLE ? WGK / 16 : 1)
        for (int k = 0; k < kn; k += 16) {
          uint32_t fa[4], fb[4];
          frag_at(fa, sX, LR, (t / NP) * 16, k);
          frag_b(fb, sY, LW, (t % NP) * 16, k);
          mma_bf16(acc[u][0], fa, fb);
          mma_bf16(acc[u][1], fa, fb + 2);
        }
      }
    }
    if (sums) {
      const int at = (i * WGK) % CSP;   // this stage's first pixel within its column sum
      if (lane_c < LANES)
#pragma unroll 8
        for (; next < at + WGK; next += LANES) {
          const float2 v = unpack_bf16(*reinterpret_cast<const uint32_t *>(sY + (next - at) * LW + col));
          csum0 += v.x;
          csum1 += v.y;
        }
      if (at + WGK == CSP) {
        if (lane_c < LANES) {
          sc[lane_c * W + col] = csum0;
          sc[lane_c * W + col + 1] = csum1;
        }
        __syncthreads();
        if (threadIdx.x < W) {
          float t = 0.f;
          for (int l = 0; l < LANES; l++) t += sc[l * W + threadIdx.x];
          sums[((p0 + (size_t)i * WGK) / CSP) * W + threadIdx.x] = t;
        }
        next = lane_c;
        csum0 = csum1 = 0.f;
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int t = warp + 8 * u;
    if (t >= units) break;
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        *reinterpret_cast<float2 *>(partial + ((size_t)blockIdx.x * R + (t / NP) * 16 + gid + 8 * h) * W + (t % NP) * 16 + c * 8 + tig * 2) =
            make_float2(acc[u][c][2 * h], acc[u][c][2 * h + 1]);
  }
}

// ---- the decoder, D1 = gelu(D0 W1 + c1), out = D1 W2 + c2, and its backward.  hidden a multiple
// of 16 up to 128, nsub up to 16 (padded with zero columns).
constexpr int DH = 128, DN = 16, DLN = DN + 8;
struct DecArgs {
  const bf16 *d0;              // [rows][W]
  const bf16 *w1, *w2;         // [W][hid], [hid][ns]
  const float *c1, *c2;
  bf16 *d1pre, *d1;            // [rows][hid]: stored by the forward pass of training (null: not), read by the backward
  float *out;                  // [rows][ns]
  const bf16 *dout;            // backward: [rows][ns]
  bf16 *dd1, *dd0;             // [rows][hid], [rows][W]
  float *dw1, *dw2;            // partial gradients per chunk of ny rows: [W][hid], [hid][ns]
  int rows, hid, ns, ny;
};
template <int W> __host__ __device__ constexpr size_t dec_fwd_smem(int hid) { return 2 * ((size_t)W * (hid + 8) + (size_t)hid * DLN + 8 * 16 * (W + 8)); }
template <int W> __host__ __device__ constexpr size_t dec_bwd_smem(int hid)
{
  return 2 * ((size_t)W * (hid + 8) + (size_t)hid * DLN + RNY * ((size_t)W + 8 + hid + 8 + DLN));
}

template <int W>
__device__ __forceinline__ void dec_weights(bf16 *sW1, bf16 *sW2, const DecArgs &a)
{
  if (a.hid == DH) copy_tile<DH>(sW1, a.hid + 8, a.w1, a.hid, W, a.hid, RT);
  else copy_tile(sW1, a.hid + 8, a.w1, a.hid, W, a.hid, RT);
  for (int e = threadIdx.x; e < a.hid * DN; e += RT) {
    const int r = e / DN, c = e - r * DN;
    sW2[r * DLN + c] = (c < a.ns) ? a.w2[r * a.ns + c] : __float2bfloat16(0.f);
  }
}

// one warp per 16 rows: the hidden values of 16 channels at a time go from the first product's
// accumulators through GELU straight into the second product's operand registers
template <int W>
__global__ void __launch_bounds__(RT, 2) dec_fwd(const DecArgs a)
{
  constexpr int LW = W + 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int LH = a.hid + 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  bf16 *sW1 = reinterpret_cast<bf16 *>(rsm), *sW2 = sW1 + W * LH, *sD = sW2 + a.hid * DLN + warp * 16 * LW;
  dec_weights<W>(sW1, sW2, a);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const bool pair = a.ns % 2 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 7) == 0;
  for (int r0 = (blockIdx.x * 8 + warp) * 16; r0 < a.rows; r0 += gridDim.x * 128) {
    for (int e = lane; e < 16 * (W / 8); e += 32) {
      const int r = min(r0 + e / (W / 8), a.rows - 1);
      cp_async16(smem_addr(sD + (e / (W / 8)) * LW + (e % (W / 8)) * 8), a.d0 + (size_t)r * W + (e % (W / 8)) * 8, 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    uint32_t fd[W / 16][4];
#pragma unroll
    for (int k = 0; k < W / 16; k++) frag_a(fd[k], sD, LW, 0, k * 16);
    float o[2][4] = {};
    for (int hc = 0; hc < a.hid; hc += 16) {
      float acc[2][4] = {};
#pragma unroll
      for (int k = 0; k < W / 16; k++) {
        uint32_t fb[4];
        frag_b(fb, sW1, LH, hc, k * 16);
        mma_bf16(acc[0], fd[k], fb);
        mma_bf16(acc[1], fd[k], fb + 2);
      }
      uint32_t fa[4], fb[4];
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = hc + t * 8 + tig * 2, r = r0 + gid + 8 * h;
          const float x = acc[t][2 * h] + a.c1[c], y = acc[t][2 * h + 1] + a.c1[c + 1];
          fa[2 * t + h] = gelu_pack(x, y);
          if (a.d1 && r < a.rows) {
            *reinterpret_cast<uint32_t *>(a.d1pre + (size_t)r * a.hid + c) = pack_bf16(x, y);
            *reinterpret_cast<uint32_t *>(a.d1 + (size_t)r * a.hid + c) = fa[2 * t + h];
          }
        }
      frag_b(fb, sW2, DLN, 0, hc);
      mma_bf16(o[0], fa, fb);
      mma_bf16(o[1], fa, fb + 2);
    }
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = t * 8 + tig * 2, r = r0 + gid + 8 * h;
        if (r >= a.rows || c >= a.ns) continue;
        float *p = a.out + (size_t)r * a.ns + c;
        const float x = o[t][2 * h] + a.c2[c];
        if (pair) *reinterpret_cast<float2 *>(p) = make_float2(x, o[t][2 * h + 1] + a.c2[c + 1]);
        else {
          p[0] = x;
          if (c + 1 < a.ns) p[1] = o[t][2 * h + 1] + a.c2[c + 1];
        }
      }
    __syncwarp();
  }
}

// one chunk of ny rows (one receiver of one sample) at a time: both weight gradients' partials,
// k over the chunk's rows ascending, and the data gradient
template <int W>
__global__ void __launch_bounds__(RT, 2) dec_bwd(const DecArgs a)
{
  constexpr int LW = W + 8;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int LH = a.hid + 8, HT = a.hid / 16, rows = (a.ny + 15) / 16 * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  bf16 *sW1 = reinterpret_cast<bf16 *>(rsm), *sW2 = sW1 + W * LH, *sD0 = sW2 + a.hid * DLN, *sD1 = sD0 + RNY * LW, *sP = sD1 + RNY * LH;
  dec_weights<W>(sW1, sW2, a);
  zero_rows(sD0, LW, a.ny, rows, RT);
  zero_rows(sD1, LH, a.ny, rows, RT);
  zero_rows(sP, DLN, a.ny, rows, RT);
  for (int u = blockIdx.x; u < a.rows / a.ny; u += gridDim.x) {
    const size_t r0 = (size_t)u * a.ny;
    copy_tile<W>(sD0, LW, a.d0 + r0 * W, W, a.ny, W, RT);
    if (a.hid == DH) copy_tile<DH>(sD1, LH, a.d1 + r0 * a.hid, a.hid, a.ny, a.hid, RT);
    else copy_tile(sD1, LH, a.d1 + r0 * a.hid, a.hid, a.ny, a.hid, RT);
    cp_async_commit();
    for (int e = threadIdx.x; e < a.ny * DN; e += RT) {
      const int r = e / DN, c = e - r * DN;
      sP[r * DLN + c] = (c < a.ns) ? a.dout[(r0 + r) * a.ns + c] : __float2bfloat16(0.f);
    }
    cp_async_wait<0>();
    __syncthreads();
    // dW2 = D1^T dout
    for (int t = warp; t < HT; t += 8) {
      float acc[2][4] = {};
      for (int k = 0; k < rows; k += 16) {
        uint32_t fa[4], fb[4];
        frag_at(fa, sD1, LH, t * 16, k);
        frag_b(fb, sP, DLN, 0, k);
        mma_bf16(acc[0], fa, fb);
        mma_bf16(acc[1], fa, fb + 2);
      }
#pragma unroll
      for (int v = 0; v < 2; v++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = t * 16 + gid + 8 * (i >> 1), c = v * 8 + tig * 2 + (i & 1);
          if (c < a.ns) a.dw2[((size_t)u * a.hid + r) * a.ns + c] = acc[v][i];
        }
    }
    __syncthreads();   // D1 has been read: its place takes dD1
    const int m0 = warp * 16;
    if (m0 < rows) {
      uint32_t fa[4];
      frag_a(fa, sP, DLN, m0, 0);
      for (int hc = 0; hc < a.hid; hc += 16) {
        float acc[2][4] = {};
        uint32_t fb[4];
        frag_bt(fb, sW2, DLN, hc, 0);
        mma_bf16(acc[0], fa, fb);
        mma_bf16(acc[1], fa, fb + 2);
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int c = hc + t * 8 + tig * 2, r = m0 + gid + 8 * h;
            if (r >= a.ny) continue;
            const size_t o = (r0 + r) * a.hid + c;
            const float2 p = unpack_bf16(*reinterpret_cast<const uint32_t *>(a.d1pre + o));
            const uint32_t d = pack_bf16(round_bf16(acc[t][2 * h]) * gelu_grad_f(p.x), round_bf16(acc[t][2 * h + 1]) * gelu_grad_f(p.y));
            *reinterpret_cast<uint32_t *>(sD1 + r * LH + c) = d;
            *reinterpret_cast<uint32_t *>(a.dd1 + o) = d;
          }
      }
    }
    __syncthreads();
    // dW1 = D0^T dD1
    for (int t = warp; t < (W / 16) * HT; t += 8) {
      const int mt = t / HT, nt = t - mt * HT;
      float acc[2][4] = {};
      for (int k = 0; k < rows; k += 16) {
        uint32_t fa[4], fb[4];
        frag_at(fa, sD0, LW, mt * 16, k);
        frag_b(fb, sD1, LH, nt * 16, k);
        mma_bf16(acc[0], fa, fb);
        mma_bf16(acc[1], fa, fb + 2);
      }
#pragma unroll
      for (int v = 0; v < 2; v++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          *reinterpret_cast<float2 *>(a.dw1 + ((size_t)u * W + mt * 16 + gid + 8 * h) * a.hid + nt * 16 + v * 8 + tig * 2) =
              make_float2(acc[v][2 * h], acc[v][2 * h + 1]);
    }
    // dD0 = dD1 W1^T
    if (m0 < rows) {
      float acc[W / 8][4] = {};
      for (int k = 0; k < a.hid; k += 16) {
        uint32_t fa[4], fb[4];
        frag_a(fa, sD1, LH, m0, k);
#pragma unroll
        for (int n = 0; n < W / 8; n += 2) {
          frag_bt(fb, sW1, LH, n * 8, k);
          mma_bf16(acc[n], fa, fb);
          mma_bf16(acc[n + 1], fa, fb + 2);
        }
      }
#pragma unroll
      for (int n = 0; n < W / 8; n++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = m0 + gid + 8 * h;
          if (r < a.ny) *reinterpret_cast<uint32_t *>(a.dd0 + (r0 + r) * W + n * 8 + tig * 2) = pack_bf16(acc[n][2 * h], acc[n][2 * h + 1]);
        }
    }
    __syncthreads();   // the tiles are free for the next chunk
  }
}

}  // namespace nnk
