// se2nn.cu -- the surrogate network runtime (include/se2nn.h): parameter and
// activation buffers, forward and backward passes as sequences of hand-written
// kernels, Adam, data-set gathers.  The Fourier layers and the decoder run as the fused
// kernels of se2nn_rows.cuh where their shapes allow (fused_ok); otherwise, and in the
// other tensor-path modes, every contraction runs through the BF16 tensor-core GEMMs of
// se2nn_gemm.cuh and se2nn_tc.cuh, with the same bits.  Everything else is a small
// elementwise, permutation or fixed-order reduction kernel below.  Results do not depend on
// scheduling: reductions are two-stage with fixed partitions, no atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <sys/mman.h>
#include <thread>
#include <unistd.h>
#include <vector>

#include "se2nn.h"
#include "se2nn_gemm.cuh"
#include "se2nn_rows.cuh"
#include "se2nn_tc.cuh"

using nnk::bf16;
using nnk::GemmArgs;

namespace {

constexpr int EW = 256;   // threads of the elementwise kernels

inline unsigned nblk(long n, int t = EW) { return (unsigned)((n + t - 1) / t); }

// ------------------------------------------------------------------ kernels
__global__ void k_f32_to_bf16(const float *x, bf16 *y, long n)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

// Wblk[mode] (2w x 2w, rows (part, ci), columns (part', co)) of the complex
// weights W = Wre + i Wim, so that [Zre Zim] Wblk = [Re(Z W) Im(Z W)]
__global__ void k_build_wblk(const float *wre, const float *wim, bf16 *blk, int nmodes, int w)
{
  const long n = (long)nmodes * 4 * w * w;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int w2 = 2 * w;
    const long mode = i / ((long)w2 * w2);
    const int r = (int)((i / w2) % w2), c = (int)(i % w2);
    const int pi = r / w, ci = r % w, po = c / w, co = c % w;
    const long o = (mode * w + ci) * w + co;
    float v;
    if (pi == po) v = wre[o];
    else v = (pi == 0) ? wim[o] : -wim[o];
    blk[i] = __float2bfloat16(v);
  }
}

// gradient of Wre, Wim from the gradient of Wblk
__global__ void k_fold_wblk(const float *dblk, float *dwre, float *dwim, int nmodes, int w)
{
  const long n = (long)nmodes * w * w;
  const int w2 = 2 * w;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const long mode = i / ((long)w * w);
    const int ci = (int)((i / w) % w), co = (int)(i % w);
    const float *d = dblk + mode * w2 * w2;
    dwre[i] = d[ci * w2 + co] + d[(w + ci) * w2 + w + co];
    dwim[i] = d[ci * w2 + w + co] - d[(w + ci) * w2 + co];
  }
}

// Z[b][j][part][kx][c]  <->  Zp[(j, kx)][b][part][c]    (dir 0: Z -> Zp, 1: Zp -> Z)
__global__ void k_permute_modes(const bf16 *src, bf16 *dst, int B, int m, int w, int dir)
{
  const int jn = 2 * m;
  const long n = (long)B * jn * 2 * m * w;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    // i indexes Z
    const int c = (int)(i % w);
    const int kx = (int)((i / w) % m);
    const int part = (int)((i / ((long)w * m)) % 2);
    const int j = (int)((i / ((long)w * m * 2)) % jn);
    const int b = (int)(i / ((long)w * m * 2 * jn));
    const long p = (((long)(j * m + kx) * B + b) * 2 + part) * w + c;
    if (dir == 0) dst[p] = src[i];
    else dst[i] = src[p];
  }
}

__global__ void k_gelu_bwd(const bf16 *dpost, const bf16 *pre, bf16 *dpre, long n)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dpre[i] = __float2bfloat16(__bfloat162float(dpost[i]) * nnk::gelu_grad_f(__bfloat162float(pre[i])));
}

// column sums of X[M][N] (bf16): partial[chunk][N] over rows [chunk*rows, ...).  With N <= EW
// the block's threads split into EW / N row lanes per column; each lane sums every
// (EW / N)-th row of the chunk and the lanes are added in lane order (fixed partition).
// The rows pass through shared memory by 16-byte copies where N allows (a lane's own
// 2-byte loads left the memory system idle: 36 us for 67 MB).
constexpr int CSE = 4096;   // elements per stage
__global__ void __launch_bounds__(EW) k_colsum_partial(const bf16 *X, long M, int N, long rows, float *partial)
{
  __shared__ float s[EW];
  __shared__ __align__(16) bf16 st[4 * CSE];
  const long r0 = blockIdx.y * rows, r1 = (r0 + rows < M) ? r0 + rows : M;
  if (N <= EW) {
    const int lanes = EW / N, c = threadIdx.x % N, lane = threadIdx.x / N;
    float v = 0.f;
    if (N % 8 == 0) {
      const int csr = CSE / N, nst = (int)((r1 - r0 + csr - 1) / csr), per = N / 8;   // rows per stage, stages
      auto load = [&](int i) {
        if (i < nst) {
          const int n = (int)min((long)csr, r1 - r0 - (long)i * csr) * per;
          const bf16 *src = X + (r0 + (long)i * csr) * N;
          for (int e = threadIdx.x; e < n; e += EW) nnk::cp_async16(nnk::smem_addr(st + (i & 3) * CSE + e * 8), src + e * 8, 16);
        }
        nnk::cp_async_commit();
      };
      for (int i = 0; i < 3; i++) load(i);
      int next = lane;   // this lane's next row of the chunk
      for (int i = 0; i < nst; i++) {
        nnk::cp_async_wait<2>();
        __syncthreads();
        load(i + 3);
        const bf16 *t = st + (i & 3) * CSE;
        const int end = (int)min((long)csr * (i + 1), r1 - r0);
        if (lane < lanes) {
#pragma unroll 8
          for (; next < end; next += lanes) v += __bfloat162float(t[(next - csr * i) * N + c]);
        }
      }
      nnk::cp_async_wait<0>();
    } else if (lane < lanes) {
      for (long r = r0 + lane; r < r1; r += lanes) v += __bfloat162float(X[r * N + c]);
    }
    s[threadIdx.x] = v;
    __syncthreads();
    if ((int)threadIdx.x < N) {
      float t = 0.f;
      for (int l = 0; l < lanes; l++) t += s[l * N + threadIdx.x];
      partial[(long)blockIdx.y * N + threadIdx.x] = t;
    }
    return;
  }
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    float t = 0.f;
    for (long r = r0; r < r1; r++) t += __bfloat162float(X[r * N + n]);
    partial[(long)blockIdx.y * N + n] = t;
  }
}

// out[i] = sum over k < nparts of partial[k][i], in order.  A block takes 32 columns: all its
// threads bring the partials into shared memory, many loads in flight, and one warp adds
// them in order there (adding straight from global memory cost one L2 round trip after
// another: 512 parts of 64 columns took 45 us)
constexpr int SPC = 32, SPK = 256;   // columns, parts per pass
// up to four sums in one launch
struct SumJob {
  const float *partial;
  float *out;
  int nparts;
  long n;
};
struct SumJobs {
  SumJob job[4];
  int first[5];   // first block of each job, and the end
};
__global__ void __launch_bounds__(EW) k_sum_parts(const SumJobs jobs)
{
  __shared__ float s[SPK][SPC];
  int which = 0;
  while ((int)blockIdx.x >= jobs.first[which + 1]) which++;
  const float *partial = jobs.job[which].partial;
  const int nparts = jobs.job[which].nparts;
  const long n = jobs.job[which].n;
  const int c = threadIdx.x % SPC, lane = threadIdx.x / SPC;
  const long i = (long)(blockIdx.x - jobs.first[which]) * SPC + c;
  float t = 0.f;
  for (int k0 = 0; k0 < nparts; k0 += SPK) {
    float v[SPK / (EW / SPC)];
#pragma unroll
    for (int u = 0; u < SPK / (EW / SPC); u++) {
      const int k = k0 + lane + u * (EW / SPC);
      v[u] = (k < nparts && i < n) ? partial[(long)k * n + i] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SPK / (EW / SPC); u++) s[lane + u * (EW / SPC)][c] = v[u];
    __syncthreads();
    if (lane == 0) {
      const int m = min(SPK, nparts - k0);
#pragma unroll 16
      for (int k = 0; k < m; k++) t += s[k][c];
    }
  }
  if (lane == 0 && i < n) jobs.job[which].out[i] = t;
}

cudaError_t sum_parts(cudaStream_t st, std::initializer_list<SumJob> list)
{
  SumJobs jobs;
  memset(&jobs, 0, sizeof(jobs));
  int k = 0, blocks = 0;
  for (const SumJob &j : list) {
    jobs.job[k] = j;
    jobs.first[k++] = blocks;
    blocks += (int)nblk(j.n, SPC);
  }
  for (; k < 5; k++) jobs.first[k] = blocks;
  k_sum_parts<<<blocks, EW, 0, st>>>(jobs);
  return cudaGetLastError();
}

// D0[((b*nrec + r)*ny + row)] = H[b][row][rec_x[r]][0:w]: every row of each receiver's column
__global__ void k_decoder_gather(const bf16 *H, const int *rec_x, int B, int nrec, int ny, int nx, int w, bf16 *D0)
{
  const long n = (long)B * nrec * ny * w;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int c = (int)(i % w);
    const long q = i / w;
    const int row = (int)(q % ny), r = (int)((q / ny) % nrec), b = (int)(q / ((long)ny * nrec));
    D0[i] = H[(((long)b * ny + row) * nx + rec_x[r]) * w + c];
  }
}

// dH[b][row][x][c] = sum over receivers r in column x of dD0[((b*nrec + r)*ny + row)][c],
// eight channels a thread (w is a multiple of 16)
__global__ void k_decoder_scatter(const bf16 *dD0, const int *rec_x, int B, int nrec, int ny, int nx, int w, bf16 *dH)
{
  const int w8 = w / 8;
  const long n = (long)B * ny * nx * w8;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int c = (int)(i % w8) * 8;
    const long pix = i / w8;
    const int x = (int)(pix % nx), row = (int)((pix / nx) % ny), b = (int)(pix / ((long)nx * ny));
    float v[8] = {};
    for (int r = 0; r < nrec; r++)
      if (rec_x[r] == x) {
        const bf16 *s = dD0 + (((long)b * nrec + r) * ny + row) * w + c;
        for (int q = 0; q < 8; q++) v[q] += __bfloat162float(s[q]);
      }
    *reinterpret_cast<uint4 *>(dH + pix * w + c) =
        make_uint4(nnk::pack_bf16(v[0], v[1]), nnk::pack_bf16(v[2], v[3]), nnk::pack_bf16(v[4], v[5]), nnk::pack_bf16(v[6], v[7]));
  }
}

// squared-error partial sums (double, per block) and dL/dout = 2 (out - t) / n
__global__ void k_mse(const float *out, const float *target, long n, double *partial, bf16 *dout)
{
  __shared__ double s[EW];
  double acc = 0.0;
  const float scale = 2.0f / (float)n;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float d = out[i] - target[i];
    acc += (double)d * (double)d;
    dout[i] = __float2bfloat16(scale * d);
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

__device__ __forceinline__ float adam_1(float p, float g, float &m, float &v, float lr, float b1, float b2, float eps, float wd,
                                        float c1, float c2)
{
  // (the roundings are spelled out: they decide which operand copies change)
  m = __fmaf_rn(1.f - b1, g, __fmul_rn(b1, m));
  v = __fmaf_rn(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, v));
  const float mh = m / c1, vh = v / c2;
  return __fmaf_rn(-lr, __fmaf_rn(wd, p, mh / (sqrtf(vh) + eps)), p);
}

// four parameters a thread (16-byte accesses); pb: the BF16 operand copy of the parameters
__global__ void k_adam(float *p, const float *g, float *m, float *v, bf16 *pb, long n, float lr, float b1, float b2,
                       float eps, float wd, float c1, float c2)
{
  const long i = 4 * (blockIdx.x * (long)blockDim.x + threadIdx.x);
  if (i + 4 <= n) {
    float4 P = *reinterpret_cast<float4 *>(p + i), M = *reinterpret_cast<float4 *>(m + i), V = *reinterpret_cast<float4 *>(v + i);
    const float4 G = *reinterpret_cast<const float4 *>(g + i);
    P.x = adam_1(P.x, G.x, M.x, V.x, lr, b1, b2, eps, wd, c1, c2);
    P.y = adam_1(P.y, G.y, M.y, V.y, lr, b1, b2, eps, wd, c1, c2);
    P.z = adam_1(P.z, G.z, M.z, V.z, lr, b1, b2, eps, wd, c1, c2);
    P.w = adam_1(P.w, G.w, M.w, V.w, lr, b1, b2, eps, wd, c1, c2);
    *reinterpret_cast<float4 *>(p + i) = P;
    *reinterpret_cast<float4 *>(m + i) = M;
    *reinterpret_cast<float4 *>(v + i) = V;
    *reinterpret_cast<uint2 *>(pb + i) = make_uint2(nnk::pack_bf16(P.x, P.y), nnk::pack_bf16(P.z, P.w));
  } else {
    for (long k = i; k < n; k++) {
      p[k] = adam_1(p[k], g[k], m[k], v[k], lr, b1, b2, eps, wd, c1, c2);
      pb[k] = __float2bfloat16(p[k]);
    }
  }
}

// network input of sample idx[b]: normalised materials, source blob, coordinates
__global__ void k_build_inputs(const float *mat, const float *src, const int *idx, int B, int ny, int nx, int cin,
                               float inv2s2, bf16 *x)
{
  const long n = (long)B * ny * nx;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;   // 16-byte stores: 51 -> 8 us for a batch of 32
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int cx = (int)(i % nx), cy = (int)((i / nx) % ny), b = (int)(i / ((long)nx * ny));
    const long s = idx[b];
    // network row cy counts down from the top surface: material row ny - 1 - cy, source row ny - y
    const float *mm = mat + ((s * ny + (ny - 1 - cy)) * nx + cx) * 3;
    const float dx = (cx + 0.5f) - src[2 * s], dy = (cy + 0.5f) - ((float)ny - src[2 * s + 1]);
    float ch[6];
    ch[0] = (mm[0] - 5000.f) * (1.f / 1500.f);   // vp
    ch[1] = (mm[1] - 2800.f) * (1.f / 800.f);    // vs
    ch[2] = (mm[2] - 2500.f) * (1.f / 500.f);    // rho
    ch[3] = __expf(-(dx * dx + dy * dy) * inv2s2);
    ch[4] = (2.f * cx + 1.f) / nx - 1.f;
    ch[5] = (2.f * cy + 1.f) / ny - 1.f;
    bf16 *o = x + i * cin;
    if (vec) {   // (cin is a multiple of 16)
      *reinterpret_cast<uint4 *>(o) = make_uint4(nnk::pack_bf16(ch[0], ch[1]), nnk::pack_bf16(ch[2], ch[3]), nnk::pack_bf16(ch[4], ch[5]), 0u);
      for (int c = 8; c < cin; c += 8) *reinterpret_cast<uint4 *>(o + c) = make_uint4(0u, 0u, 0u, 0u);
    } else {
      for (int c = 0; c < cin; c++) o[c] = __float2bfloat16(c < 6 ? ch[c] : 0.f);
    }
  }
}

__global__ void k_gather_rows(const float *src, const int *idx, int B, long row, float *dst)
{
  const long n = (long)B * row;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = src[(long)idx[i / row] * row + i % row];
}

}  // namespace

// ------------------------------------------------------------------ the network
struct se2nn {
  se2nn_config c{};
  int npix = 0, w = 0, m = 0, nmodes = 0, L = 0;
  long P = 0;
  // parameter offsets (floats)
  long oW0 = 0, ob0 = 0, oW1 = 0, oc1 = 0, oW2 = 0, oc2 = 0;
  std::vector<long> oWre, oWim, oW, ob;
  float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  long adam_t = 0;
  // BF16 copy of all parameters, and into it the matrices the kernels read; the 2w x 2w mode
  // blocks of the GEMM path are formed when that path next runs or, once it has been captured,
  // with every change of the parameters (the captured pass reads them when it is replayed)
  bf16 *Pb = nullptr, *W0b = nullptr, *W1b = nullptr, *W2b = nullptr;
  std::vector<bf16 *> Wb, Wreb, Wimb, Wblk;
  bool wblk_stale = true, wblk_captured = false;
  int nsm = 0, row_ctas[4] = {1, 1, 1, 1};   // SMs; the row kernels' resident CTAs per SM
  // DFT matrices (BF16): Ex [2m][nx], My [4m][2ny], Myinv [2ny][4m] (= My^T), Exinv [nx][2m],
  // and the transposes ExT [nx][2m], ExinvT [2m][nx]
  bf16 *Ex = nullptr, *My = nullptr, *Myinv = nullptr, *Exinv = nullptr, *ExT = nullptr, *ExinvT = nullptr;
  int *rec_x = nullptr;
  float *lut = nullptr;   // GELU' at BF16 arguments
  // activations (max batch)
  std::vector<bf16 *> H, Apre, Zp;
  bf16 *S = nullptr, *Xf = nullptr, *Z = nullptr, *Yp = nullptr, *Y = nullptr, *Yy = nullptr, *dZp = nullptr;
  bf16 *D0 = nullptr, *D1pre = nullptr, *D1 = nullptr, *dpred = nullptr;
  bf16 *dHa = nullptr, *dHb = nullptr, *dA = nullptr, *dD1 = nullptr, *dD0 = nullptr;
  float *out = nullptr, *partial = nullptr, *colpart = nullptr, *decpart = nullptr, *dblk = nullptr;
  double *lpart = nullptr;
  long partial_n = 0;
  int split = 1, nsub = 1;
  cudaStream_t stream = nullptr;
  std::vector<void *> allocs;
  char err[512] = {0};
};

namespace {

thread_local char g_nn_create_err[512];

int nfail(se2nn *h, int code, const char *fmt, ...)
{
  char *buf = h ? h->err : g_nn_create_err;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, 512, fmt, ap);
  va_end(ap);
  return code;
}

#define NCK(h, call)                                                                                             \
  do {                                                                                                           \
    cudaError_t e_ = (call);                                                                                     \
    if (e_ != cudaSuccess) return nfail((h), -2, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

template <class T>
int nalloc(se2nn *h, T **p, size_t count)
{
  *p = nullptr;
  void *q = nullptr;
  cudaError_t e = cudaMalloc(&q, count ? count * sizeof(T) : 16);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nfail(h, -3, "cudaMalloc(%zu bytes): %s", count * sizeof(T), cudaGetErrorString(e));
  }
  h->allocs.push_back(q);
  *p = static_cast<T *>(q);
  return 0;
}

uint64_t mix64(uint64_t *s)
{
  uint64_t z = (*s += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

float uniform_pm(uint64_t *s, float a) { return a * (float)(2.0 * ((double)(mix64(s) >> 11) / 9007199254740992.0) - 1.0); }

int upload_bf16(se2nn *h, bf16 *dst, const std::vector<float> &src)
{
  std::vector<bf16> t(src.size());
  for (size_t i = 0; i < src.size(); i++) t[i] = __float2bfloat16(src[i]);
  NCK(h, cudaMemcpy(dst, t.data(), t.size() * sizeof(bf16), cudaMemcpyHostToDevice));
  return 0;
}

// the truncated DFT matrices of the spectral layers (built in double, stored BF16)
int build_dft(se2nn *h)
{
  const int nx = h->c.nx, ny = h->c.ny, m = h->m;
  const double tau = 2.0 * M_PI;
  auto ky_of = [&](int j) { return j < m ? j : ny - 2 * m + j; };
  std::vector<float> ex(2 * m * nx), my(4 * m * 2 * ny), myi(2 * ny * 4 * m), exi(nx * 2 * m), ext(nx * 2 * m), exit(2 * m * nx);
  for (int kx = 0; kx < m; kx++)
    for (int x = 0; x < nx; x++) {
      const double t = tau * kx * x / nx;
      ex[(0 * m + kx) * nx + x] = (float)cos(t);
      ex[(1 * m + kx) * nx + x] = (float)-sin(t);
      const double wk = (kx == 0 ? 1.0 : 2.0) / ((double)nx * ny);
      exi[x * 2 * m + 0 * m + kx] = (float)(wk * cos(t));
      exi[x * 2 * m + 1 * m + kx] = (float)(-wk * sin(t));
    }
  for (int j = 0; j < 2 * m; j++)
    for (int y = 0; y < ny; y++) {
      const double t = tau * ky_of(j) * y / ny, c = cos(t), s = sin(t);
      // forward: Z = sum_y e^{-i t} Xf
      my[(j * 2 + 0) * 2 * ny + y * 2 + 0] = (float)c;
      my[(j * 2 + 0) * 2 * ny + y * 2 + 1] = (float)s;
      my[(j * 2 + 1) * 2 * ny + y * 2 + 0] = (float)-s;
      my[(j * 2 + 1) * 2 * ny + y * 2 + 1] = (float)c;
      // inverse: Yy = sum_j e^{+i t} Y
      myi[(y * 2 + 0) * 4 * m + j * 2 + 0] = (float)c;
      myi[(y * 2 + 0) * 4 * m + j * 2 + 1] = (float)-s;
      myi[(y * 2 + 1) * 4 * m + j * 2 + 0] = (float)s;
      myi[(y * 2 + 1) * 4 * m + j * 2 + 1] = (float)c;
    }
  for (int k = 0; k < 2 * m; k++)
    for (int x = 0; x < nx; x++) {
      ext[x * 2 * m + k] = ex[k * nx + x];
      exit[k * nx + x] = exi[x * 2 * m + k];
    }
  // one allocation and one copy of all six, each on a 256-byte boundary
  struct { const std::vector<float> &v; bf16 **p; } parts[] = {{ext, &h->ExT}, {exit, &h->ExinvT}, {ex, &h->Ex},
                                                               {my, &h->My}, {myi, &h->Myinv}, {exi, &h->Exinv}};
  auto padded = [](size_t n) { return (n + 127) / 128 * 128; };
  std::vector<float> all;
  for (auto &q : parts) {
    all.insert(all.end(), q.v.begin(), q.v.end());
    all.resize(padded(all.size()));
  }
  bf16 *at = nullptr;
  int rc;
  if ((rc = nalloc(h, &at, all.size())) || (rc = upload_bf16(h, at, all))) return rc;
  for (auto &q : parts) {
    *q.p = at;
    at += padded(q.v.size());
  }
  return 0;
}

bool capturing(const se2nn *h)
{
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->stream, &st) != cudaSuccess) cudaGetLastError();
  return st != cudaStreamCaptureStatusNone;
}

// the mode blocks of the GEMM path, from the parameters
int build_wblk(se2nn *h)
{
  for (int l = 0; l < h->L; l++)
    k_build_wblk<<<nblk((long)h->nmodes * 4 * h->w * h->w), EW, 0, h->stream>>>(h->params + h->oWre[l], h->params + h->oWim[l],
                                                                                h->Wblk[l], h->nmodes, h->w);
  NCK(h, cudaGetLastError());
  return 0;
}

// after each change of the parameters.  What is captured has not run: it takes the blocks along and
// leaves the flag.
int params_changed(se2nn *h)
{
  const bool cap = capturing(h), build = h->wblk_captured || cap;
  if (!cap) h->wblk_stale = !build;
  return build ? build_wblk(h) : 0;
}

// before the GEMM path reads the blocks
int need_wblk(se2nn *h)
{
  if (capturing(h)) {
    h->wblk_captured = true;
    return h->wblk_stale ? build_wblk(h) : 0;
  }
  if (!h->wblk_stale) return 0;
  h->wblk_stale = false;
  return build_wblk(h);
}

// refresh the BF16 operand copy from the FP32 master parameters
int refresh_bf16(se2nn *h)
{
  k_f32_to_bf16<<<nblk(h->P), EW, 0, h->stream>>>(h->params, h->Pb, h->P);
  NCK(h, cudaGetLastError());
  return params_changed(h);
}

}  // namespace

namespace {

GemmArgs mk(const bf16 *A, long lda, long sA, int tA, const bf16 *B, long ldb, long sB, int tB, int M, int N, int K,
            int batch, void *C, long ldc, long sC, int c_f32)
{
  GemmArgs g;
  memset(&g, 0, sizeof(g));
  g.A = A; g.lda = lda; g.sA = sA; g.transA = tA;
  g.B = B; g.ldb = ldb; g.sB = sB; g.transB = tB;
  g.M = M; g.N = N; g.K = K; g.batch = batch;
  g.alpha = 1.f; g.beta = 0.f;
  g.C = C; g.ldc = ldc; g.sC = sC; g.c_f32 = c_f32;
  return g;
}

// ---- the tensor-core (tcgen05) path for the row GEMMs -----------------------------
// 0: every GEMM runs gemm_bf16; 1 (default): qualifying row GEMMs run gemm_tc except those
// with N <= 64 and 32 < K <= 64 (the 1x1 convolutions and their data gradients, where
// the mma.sync kernel measured faster); 2: every qualifying row GEMM runs gemm_tc
std::atomic<int> g_tc_path{1};
std::atomic<long> g_tc_launches{0}, g_mma_launches{0};
__device__ int g_tc_err;

bool tc_eligible(const GemmArgs &g)
{
  return g_tc_path && (g_tc_path == 2 || !(g.N <= 64 && g.K > 32 && g.K <= 64)) && !g.transA && g.batch == 1 && g.M >= nnk::TC_M && g.K % 16 == 0 && g.K >= 16 &&
         g.K <= nnk::TC_KMAX && g.N % 16 == 0 && g.N >= 16 && g.N <= nnk::TC_NMAX && g.lda % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(g.A) & 15) == 0;
}

// per device (the current one at the launch): the error flag's address, the SM count and
// the kernel's shared-memory limit, set up on the first launch on that device
struct TcDevice {
  int *err = nullptr;
  int nsm = 0;
};

cudaError_t launch_gemm_tc(const GemmArgs &g, cudaStream_t st)
{
  static std::mutex mu;
  static TcDevice devs[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  TcDevice d;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!devs[dev].err) {
      int nsm = 0;
      int *err = nullptr;
      e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess) e = cudaGetSymbolAddress((void **)&err, g_tc_err);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(nnk::gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)nnk::tc_smem_bytes(nnk::TC_NMAX, nnk::TC_KMAX));
      if (e != cudaSuccess) return e;
      devs[dev].nsm = nsm;
      devs[dev].err = err;
    }
    d = devs[dev];
  }
  int *err = d.err;
  const int nsm = d.nsm;
  // resident CTAs per SM: what registers and shared memory allow, capped by the 512
  // tensor-memory columns of an SM (a CTA beyond them would wait in its allocation)
  const size_t smem = nnk::tc_smem_bytes(g.N, g.K);
  int occ = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, nnk::gemm_tc, nnk::TC_THREADS, smem) != cudaSuccess) {
    cudaGetLastError();
    occ = 1;
  }
  occ = std::max(1, std::min(occ, 512 / nnk::tc_tmem_cols(g.N)));
  const int ntiles = (g.M + nnk::TC_M - 1) / nnk::TC_M;
  const int grid = std::min(ntiles, occ * nsm);
  nnk::gemm_tc<<<grid, nnk::TC_THREADS, smem, st>>>(g, err);
  g_tc_launches++;
  return cudaGetLastError();
}

cudaError_t launch_gemm(const GemmArgs &g, cudaStream_t st)
{
  if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return cudaSuccess;
  if (tc_eligible(g)) return launch_gemm_tc(g, st);
  g_mma_launches++;
  const unsigned gy = (unsigned)((g.M + nnk::GBM - 1) / nnk::GBM), gx = (unsigned)((g.N + nnk::GBN - 1) / nnk::GBN);
  if (gy > 65535u || g.batch > 65535) return cudaErrorInvalidConfiguration;
  nnk::gemm_bf16<<<dim3(gx, gy, (unsigned)g.batch), nnk::GTHREADS, 0, st>>>(g);
  return cudaGetLastError();
}

#define GEMM(h, g) NCK((h), launch_gemm((g), (h)->stream))

// column sums of X[M][N] (bf16) into out (f32), fixed partition of rows
int colsum(se2nn *h, const bf16 *X, long M, int N, long rows, float *out)
{
  const int chunks = (int)((M + rows - 1) / rows);
  k_colsum_partial<<<dim3(1, chunks), EW, 0, h->stream>>>(X, M, N, rows, h->partial);
  NCK(h, sum_parts(h->stream, {{h->partial, out, chunks, N}}));
  return 0;
}

// out (rows x w, f32) = X^T dY over B*npix pixels, split into B*split chunks then summed in order
int weight_grad(se2nn *h, const bf16 *X, int rows, const bf16 *dY, int B, float *out)
{
  const int w = h->w, s = h->split;
  const long kc = h->npix / s;
  GemmArgs g = mk(X, rows, kc * rows, 1, dY, w, kc * w, 0, rows, w, (int)kc, B * s, h->partial, w, (long)rows * w, 1);
  GEMM(h, g);
  NCK(h, sum_parts(h->stream, {{h->partial, out, B * s, (long)rows * w}}));
  return 0;
}

// out (M x N, f32) = X^T dY for X [K][M], dY [K][N] (bf16, K rows a multiple of chunk), split-K in fixed order
int splitk_grad(se2nn *h, const bf16 *X, int M, const bf16 *dY, int N, long K, long chunk, float *out)
{
  const int parts = (int)(K / chunk);
  GemmArgs g = mk(X, M, chunk * M, 1, dY, N, chunk * N, 0, M, N, (int)chunk, parts, h->partial, N, (long)M * N, 1);
  GEMM(h, g);
  NCK(h, sum_parts(h->stream, {{h->partial, out, parts, (long)M * N}}));
  return 0;
}

// S = spectral convolution of Hin with layer l's weights; the mode-major input is kept in Zp[l]
int spectral_fwd(se2nn *h, int l, const bf16 *Hin, int B, bf16 *Sout)
{
  const int nx = h->c.nx, ny = h->c.ny, m = h->m, w = h->w;
  const long mw = (long)m * w;
  GEMM(h, mk(h->Ex, nx, 0, 0, Hin, w, (long)nx * w, 0, 2 * m, w, nx, B * ny, h->Xf, w, 2L * m * w, 0));
  GEMM(h, mk(h->My, 2 * ny, 0, 0, h->Xf, mw, (long)ny * 2 * mw, 0, 4 * m, (int)mw, 2 * ny, B, h->Z, mw, 4 * m * mw, 0));
  k_permute_modes<<<nblk((long)B * 4 * m * mw), EW, 0, h->stream>>>(h->Z, h->Zp[l], B, m, w, 0);
  GEMM(h, mk(h->Zp[l], 2 * w, (long)B * 2 * w, 0, h->Wblk[l], 2 * w, 4L * w * w, 0, B, 2 * w, 2 * w, h->nmodes, h->Yp,
             2 * w, (long)B * 2 * w, 0));
  k_permute_modes<<<nblk((long)B * 4 * m * mw), EW, 0, h->stream>>>(h->Yp, h->Y, B, m, w, 1);
  GEMM(h, mk(h->Myinv, 4 * m, 0, 0, h->Y, mw, 4 * m * mw, 0, 2 * ny, (int)mw, 4 * m, B, h->Yy, mw, 2L * ny * mw, 0));
  GEMM(h, mk(h->Exinv, 2 * m, 0, 0, h->Yy, w, 2L * m * w, 0, nx, w, 2 * m, B * ny, Sout, w, (long)nx * w, 0));
  return 0;
}

// backward of spectral_fwd: dS -> weight gradients of layer l, dHacc += dHin
int spectral_bwd(se2nn *h, int l, const bf16 *dS, int B, bf16 *dHacc)
{
  const int nx = h->c.nx, ny = h->c.ny, m = h->m, w = h->w;
  const long mw = (long)m * w;
  GEMM(h, mk(h->Exinv, 2 * m, 0, 1, dS, w, (long)nx * w, 0, 2 * m, w, nx, B * ny, h->Yy, w, 2L * m * w, 0));
  GEMM(h, mk(h->Myinv, 4 * m, 0, 1, h->Yy, mw, 2L * ny * mw, 0, 4 * m, (int)mw, 2 * ny, B, h->Y, mw, 4 * m * mw, 0));
  k_permute_modes<<<nblk((long)B * 4 * m * mw), EW, 0, h->stream>>>(h->Y, h->Yp, B, m, w, 0);
  GEMM(h, mk(h->Zp[l], 2 * w, (long)B * 2 * w, 1, h->Yp, 2 * w, (long)B * 2 * w, 0, 2 * w, 2 * w, B, h->nmodes, h->dblk,
             2 * w, 4L * w * w, 1));
  k_fold_wblk<<<nblk((long)h->nmodes * w * w), EW, 0, h->stream>>>(h->dblk, h->grads + h->oWre[l], h->grads + h->oWim[l],
                                                                    h->nmodes, w);
  GEMM(h, mk(h->Yp, 2 * w, (long)B * 2 * w, 0, h->Wblk[l], 2 * w, 4L * w * w, 1, B, 2 * w, 2 * w, h->nmodes, h->dZp,
             2 * w, (long)B * 2 * w, 0));
  k_permute_modes<<<nblk((long)B * 4 * m * mw), EW, 0, h->stream>>>(h->dZp, h->Z, B, m, w, 1);
  GEMM(h, mk(h->My, 2 * ny, 0, 1, h->Z, mw, 4 * m * mw, 0, 2 * ny, (int)mw, 4 * m, B, h->Xf, mw, 2L * ny * mw, 0));
  GemmArgs g = mk(h->Ex, nx, 0, 1, h->Xf, w, 2L * m * w, 0, nx, w, 2 * m, B * ny, dHacc, w, (long)nx * w, 0);
  g.beta = 1.f; g.Cin = dHacc; g.ldcin = w; g.sCin = (long)nx * w;
  GEMM(h, g);
  return 0;
}

// ---- the fused path (se2nn_rows.cuh): the default wherever its shapes allow; the GEMM path
// serves the others and, with se2nn_set_tensor_path 0 or 2, every shape.  Same bits.
bool fused_shape(const se2nn *h)
{
  const se2nn_config &c = h->c;
  return (h->w == 16 || h->w == 32 || h->w == 48 || h->w == 64) && c.cin <= 64 && c.nx % 16 == 0 &&
         c.nx <= nnk::RNX && c.ny % 8 == 0 && c.ny <= nnk::RNY && h->m <= nnk::RM && c.nrec <= nnk::RREC;
}
bool fused_ok(const se2nn *h, const void *x)
{
  return g_tc_path == 1 && fused_shape(h) && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
}

// Kernel set-up at create: shared-memory limits (at the largest size any network uses, so that
// handles of different shapes agree on them) and the row kernels' resident CTAs.
template <class F>
cudaError_t allow_smem(F *fn, size_t smem)
{
  return (smem > 48 * 1024) ? cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
}

template <int W, int KIND>
cudaError_t row_setup(se2nn *h)
{
  typedef nnk::RowSmem<W, KIND> S;
  cudaError_t e = allow_smem(nnk::row_kernel<W, KIND>, S::bytes(nnk::RNX, 64));
  int n = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, nnk::row_kernel<W, KIND>, nnk::RT, S::bytes(h->c.nx, h->c.cin));
  h->row_ctas[KIND] = std::max(1, n);
  return e;
}

template <int W>
int fused_setup_w(se2nn *h)
{
  cudaError_t e = row_setup<W, nnk::ROW_LIFT>(h);
  if (e == cudaSuccess) e = row_setup<W, nnk::ROW_FWD>(h);
  if (e == cudaSuccess) e = row_setup<W, nnk::ROW_BWD>(h);
  if (e == cudaSuccess) e = row_setup<W, nnk::ROW_TOP>(h);
  if (e == cudaSuccess) e = allow_smem(nnk::y_analysis<W>, nnk::y_analysis_smem(nnk::RNY));
  if (e == cudaSuccess) e = allow_smem(nnk::y_synthesis<W>, nnk::y_synthesis_smem(nnk::RNY));
  if (e == cudaSuccess) e = allow_smem(nnk::last_kernel<W>, nnk::last_smem<W>());
  if (e == cudaSuccess) e = allow_smem(nnk::mode_mix<W>, nnk::mode_smem<W>());
  if (e == cudaSuccess) e = allow_smem(nnk::mode_grad<W>, nnk::mode_grad_smem<W>());
  if (e == cudaSuccess) e = allow_smem(nnk::weight_grad_partial<W, 0, false>, nnk::wgrad_smem<W>(64));
  if (e == cudaSuccess) e = allow_smem(nnk::weight_grad_partial<W, W, true>, nnk::wgrad_smem<W>(64));
  if (e == cudaSuccess) e = allow_smem(nnk::weight_grad_partial<W, 0, true>, nnk::wgrad_smem<W>(64));
  if (e == cudaSuccess) e = allow_smem(nnk::dec_fwd<W>, nnk::dec_fwd_smem<W>(nnk::DH));
  if (e == cudaSuccess) e = allow_smem(nnk::dec_bwd<W>, nnk::dec_bwd_smem<W>(nnk::DH));
  NCK(h, e);
  return 0;
}

template <int W, int KIND>
int row_launch(se2nn *h, const nnk::RowArgs &a)
{
  nnk::row_kernel<W, KIND><<<std::min(a.rows, h->row_ctas[KIND] * h->nsm), nnk::RT, nnk::RowSmem<W, KIND>::bytes(a.nx, a.cin), h->stream>>>(a);
  NCK(h, cudaGetLastError());
  return 0;
}

// f<W>(h, ...) for the network's width
#define NN_WIDTH(f, ...)                       \
  switch (h->w) {                              \
    case 16: return f<16>(__VA_ARGS__);        \
    case 32: return f<32>(__VA_ARGS__);        \
    case 48: return f<48>(__VA_ARGS__);        \
    default: return f<64>(__VA_ARGS__);        \
  }

int fused_setup(se2nn *h)
{
  if (!fused_shape(h)) return 0;
  int rc = nalloc(h, &h->lut, nnk::GLUT);
  if (rc) return rc;
  nnk::gelu_lut_kernel<<<nblk(nnk::GLUT), EW, 0, h->stream>>>(h->lut);
  NCK(h, cudaGetLastError());
  NN_WIDTH(fused_setup_w, h)
}

nnk::RowArgs row_args(se2nn *h, int B)
{
  nnk::RowArgs a;
  memset(&a, 0, sizeof(a));
  a.rows = B * h->c.ny; a.nx = h->c.nx; a.ny = h->c.ny; a.m2 = 2 * h->m; a.cin = h->c.cin;
  a.nrec = h->c.nrec; a.rec_x = h->rec_x; a.lut = h->lut;
  return a;
}

template <int W>
int y_analysis_w(se2nn *h, const bf16 *spec, bf16 *Zp, int B)
{
  const size_t smem = nnk::y_analysis_smem(h->c.ny);
  nnk::y_analysis<W><<<dim3((h->m * W + nnk::YN - 1) / nnk::YN, B), nnk::RT, smem, h->stream>>>(nnk::YArgs{h->My, spec, Zp, h->c.ny, h->m, B});
  NCK(h, cudaGetLastError());
  return 0;
}
int y_analysis(se2nn *h, const bf16 *spec, bf16 *Zp, int B) { NN_WIDTH(y_analysis_w, h, spec, Zp, B) }

template <int W>
int y_synthesis_w(se2nn *h, const bf16 *Y, bf16 *spec, int B)
{
  const size_t smem = nnk::y_synthesis_smem(h->c.ny);
  nnk::y_synthesis<W><<<dim3((h->m * W + nnk::YN - 1) / nnk::YN, B), nnk::RT, smem, h->stream>>>(nnk::YArgs{h->Myinv, Y, spec, h->c.ny, h->m, B});
  NCK(h, cudaGetLastError());
  return 0;
}
int y_synthesis(se2nn *h, const bf16 *Y, bf16 *spec, int B) { NN_WIDTH(y_synthesis_w, h, Y, spec, B) }

template <int W>
int mode_mix(se2nn *h, int l, int B)
{
  constexpr size_t smem = nnk::mode_smem<W>();
  nnk::mode_mix<W><<<h->nmodes, nnk::RT, smem, h->stream>>>(
      nnk::ModeArgs{h->Zp[l], h->Wreb[l], h->Wimb[l], h->Y, nullptr, nullptr, nullptr, h->m, B});
  NCK(h, cudaGetLastError());
  return 0;
}

// from the spectrum rows Xf of H[l] to the spectrum rows Yy of the layer's spectral part
int spectrum_fwd(se2nn *h, int l, int B)
{
  auto mix = [&]() -> int { NN_WIDTH(mode_mix, h, l, B) };
  int rc;
  if ((rc = y_analysis(h, h->Xf, h->Zp[l], B)) || (rc = mix()) || (rc = y_synthesis(h, h->Y, h->Yy, B))) return rc;
  return 0;
}

template <int W>
int last_rows(se2nn *h, int B)
{
  const int l = h->L - 1;
  constexpr size_t smem = nnk::last_smem<W>();
  nnk::LastArgs a{h->H[l], h->Yy, h->Wb[l], h->Exinv, h->params + h->ob[l], h->rec_x, h->D0, B * h->c.ny, h->c.nx, h->c.ny,
                  2 * h->m, h->c.nrec};
  nnk::last_kernel<W><<<(a.rows + 7) / 8, nnk::RT, smem, h->stream>>>(a);
  NCK(h, cudaGetLastError());
  return 0;
}

// the lift and the Fourier layers to the decoder's input D0; keep: store the pre-activations
template <int W>
int layers_fwd(se2nn *h, const bf16 *x, int B, bool keep)
{
  int rc;
  nnk::RowArgs a = row_args(h, B);
  a.in = x; a.wt = h->W0b; a.bias = h->params + h->ob0; a.efwd = h->Ex; a.out = h->H[0]; a.spec_out = h->Xf;
  if ((rc = row_launch<W, nnk::ROW_LIFT>(h, a))) return rc;
  for (int l = 0; l < h->L; l++) {
    if ((rc = spectrum_fwd(h, l, B))) return rc;
    if (l == h->L - 1) break;
    a = row_args(h, B);
    a.in = h->H[l]; a.spec = h->Yy; a.wt = h->Wb[l]; a.bias = h->params + h->ob[l]; a.einv = h->Exinv; a.efwd = h->Ex;
    a.out = h->H[l + 1]; a.aux = keep ? h->Apre[l] : nullptr; a.spec_out = h->Xf;
    if ((rc = row_launch<W, nnk::ROW_FWD>(h, a))) return rc;
  }
  return last_rows<W>(h, B);
}

int layers_fused(se2nn *h, const bf16 *x, int B, bool keep) { NN_WIDTH(layers_fwd, h, x, B, keep) }

template <int W>
int mode_grad(se2nn *h, int l, int B)
{
  constexpr size_t smem = nnk::mode_grad_smem<W>();
  nnk::mode_grad<W><<<h->nmodes, nnk::RT, smem, h->stream>>>(
      nnk::ModeArgs{h->Zp[l], h->Wreb[l], h->Wimb[l], h->Y, h->Yp, h->grads + h->oWre[l], h->grads + h->oWim[l], h->m, B});
  NCK(h, cudaGetLastError());
  return 0;
}

// weight and bias gradients of a 1x1 convolution: X^T dY and the column sums of dY
template <int W>
int conv_grads(se2nn *h, const bf16 *X, int R, const bf16 *dY, int B, float *dw, float *db)
{
  const int kc = h->npix / h->split;
  const long rows = (long)B * h->npix;
  const bool sums = kc % nnk::CSP == 0;   // whole column sums per chunk; else a pass of their own
  auto fn = (kc % nnk::WGK) ? nnk::weight_grad_partial<W, 0, false>
            : (R == W) ? nnk::weight_grad_partial<W, W, true>
                       : nnk::weight_grad_partial<W, 0, true>;
  fn<<<B * h->split, nnk::RT, nnk::wgrad_smem<W>(R), h->stream>>>(X, R, dY, kc, h->partial, sums ? h->colpart : nullptr);
  NCK(h, cudaGetLastError());
  const SumJob w{h->partial, dw, B * h->split, (long)R * W};
  if (sums) {
    NCK(h, sum_parts(h->stream, {w, {h->colpart, db, (int)(rows / nnk::CSP), W}}));
    return 0;
  }
  NCK(h, sum_parts(h->stream, {w}));
  return colsum(h, dY, rows, W, nnk::CSP, db);
}

// backward of the Fourier layers and the lift from dD0.  dHa and dHb take turns as the layers'
// gradients: dA of layer l (below the first layer dH[0]) with its spectrum rows in Xf.
template <int W>
int layers_bwd(se2nn *h, const bf16 *x, int B)
{
  int rc;
  nnk::RowArgs a = row_args(h, B);
  a.dd0 = h->dD0; a.efwd = h->ExinvT; a.out = h->dHa; a.spec_out = h->Xf;
  if ((rc = row_launch<W, nnk::ROW_TOP>(h, a))) return rc;
  for (int l = h->L - 1; l >= 0; l--) {
    if ((rc = conv_grads<W>(h, h->H[l], W, h->dHa, B, h->grads + h->oW[l], h->grads + h->ob[l]))) return rc;
    if ((rc = y_analysis(h, h->Xf, h->Yp, B)) || (rc = mode_grad<W>(h, l, B)) || (rc = y_synthesis(h, h->Y, h->Yy, B))) return rc;
    a = row_args(h, B);
    a.in = h->dHa; a.spec = h->Yy; a.wt = h->Wb[l]; a.einv = h->ExT; a.efwd = h->ExinvT; a.out = h->dHb;
    a.pre = l ? h->Apre[l - 1] : nullptr;
    a.spec_out = l ? h->Xf : nullptr;
    if ((rc = row_launch<W, nnk::ROW_BWD>(h, a))) return rc;
    std::swap(h->dHa, h->dHb);
  }
  return conv_grads<W>(h, x, h->c.cin, h->dHa, B, h->grads + h->oW0, h->grads + h->ob0);
}

int layers_bwd_fused(se2nn *h, const bf16 *x, int B) { NN_WIDTH(layers_bwd, h, x, B) }

// ---- the fused decoder
bool fused_decoder(const se2nn *h) { return h->c.hidden <= nnk::DH && h->nsub <= nnk::DN; }

nnk::DecArgs dec_args(se2nn *h, int B)
{
  nnk::DecArgs a;
  memset(&a, 0, sizeof(a));
  a.d0 = h->D0; a.w1 = h->W1b; a.w2 = h->W2b; a.c1 = h->params + h->oc1; a.c2 = h->params + h->oc2;
  a.rows = B * h->c.nrec * h->c.ny; a.hid = h->c.hidden; a.ns = h->nsub; a.ny = h->c.ny;
  return a;
}

template <int W>
int decoder_fwd_w(se2nn *h, int B, float *out, bool keep)
{
  nnk::DecArgs a = dec_args(h, B);
  a.out = out;
  if (keep) { a.d1pre = h->D1pre; a.d1 = h->D1; }
  nnk::dec_fwd<W><<<std::min((a.rows + 127) / 128, 4 * h->nsm), nnk::RT, nnk::dec_fwd_smem<W>(a.hid), h->stream>>>(a);
  NCK(h, cudaGetLastError());
  return 0;
}
int decoder_fwd(se2nn *h, int B, float *out, bool keep) { NN_WIDTH(decoder_fwd_w, h, B, out, keep) }

// weight gradients' partials (then summed), bias gradients, dD0
template <int W>
int decoder_bwd_w(se2nn *h, int B)
{
  nnk::DecArgs a = dec_args(h, B);
  const int units = B * h->c.nrec;
  a.d1pre = h->D1pre; a.d1 = h->D1; a.dout = h->dpred; a.dd1 = h->dD1; a.dd0 = h->dD0;
  a.dw1 = h->partial; a.dw2 = h->decpart;
  nnk::dec_bwd<W><<<std::min(units, 2 * h->nsm), nnk::RT, nnk::dec_bwd_smem<W>(a.hid), h->stream>>>(a);
  const int chunks = (a.rows + 255) / 256;
  float *c2 = h->decpart + (size_t)units * a.hid * a.ns, *c1 = c2 + (size_t)chunks * a.ns;
  k_colsum_partial<<<dim3(1, chunks), EW, 0, h->stream>>>(h->dpred, a.rows, a.ns, 256, c2);
  k_colsum_partial<<<dim3(1, chunks), EW, 0, h->stream>>>(h->dD1, a.rows, a.hid, 256, c1);
  NCK(h, cudaGetLastError());
  NCK(h, sum_parts(h->stream, {{h->partial, h->grads + h->oW1, units, (long)W * a.hid},
                               {h->decpart, h->grads + h->oW2, units, (long)a.hid * a.ns},
                               {c2, h->grads + h->oc2, chunks, a.ns},
                               {c1, h->grads + h->oc1, chunks, a.hid}}));
  return 0;
}
int decoder_bwd(se2nn *h, int B) { NN_WIDTH(decoder_bwd_w, h, B) }

// keep: the pass is followed by backward (pre-activations are stored)
int forward(se2nn *h, const bf16 *x, int B, float *out, bool keep)
{
  const int w = h->w, L = h->L, nrec = h->c.nrec, hid = h->c.hidden;
  const long rows = (long)B * h->npix;
  int rc;
  const bool fused = fused_ok(h, x);
  if (fused) {
    if ((rc = layers_fused(h, x, B, keep))) return rc;
  } else {
  if ((rc = need_wblk(h))) return rc;
  {
    GemmArgs g = mk(x, h->c.cin, 0, 0, h->W0b, w, 0, 0, (int)rows, w, h->c.cin, 1, h->H[0], w, 0, 0);
    g.bias = h->params + h->ob0;
    GEMM(h, g);
  }
  for (int l = 0; l < L; l++) {
    if ((rc = spectral_fwd(h, l, h->H[l], B, h->S))) return rc;
    GemmArgs g = mk(h->H[l], w, 0, 0, h->Wb[l], w, 0, 0, (int)rows, w, w, 1, h->H[l + 1], w, 0, 0);
    g.beta = 1.f; g.Cin = h->S; g.ldcin = w;
    g.bias = h->params + h->ob[l];
    if (l < L - 1) { g.act = 1; g.aux = h->Apre[l]; g.ldaux = w; }
    GEMM(h, g);
  }
  }
  const bf16 *HL = h->H[L];
  const long drows = (long)B * nrec * h->c.ny;
  if (fused && fused_decoder(h)) return decoder_fwd(h, B, out, keep);
  if (!fused) k_decoder_gather<<<nblk(drows * w), EW, 0, h->stream>>>(HL, h->rec_x, B, nrec, h->c.ny, h->c.nx, w, h->D0);
  {
    GemmArgs g = mk(h->D0, w, 0, 0, h->W1b, hid, 0, 0, (int)drows, hid, w, 1, h->D1, hid, 0, 0);
    g.bias = h->params + h->oc1; g.act = 1; g.aux = h->D1pre; g.ldaux = hid;
    GEMM(h, g);
  }
  {
    GemmArgs g = mk(h->D1, hid, 0, 0, h->W2b, h->nsub, 0, 0, (int)drows, h->nsub, hid, 1, out, h->nsub, 0, 1);
    g.bias = h->params + h->oc2;
    GEMM(h, g);
  }
  NCK(h, cudaGetLastError());
  return 0;
}

int backward(se2nn *h, const bf16 *x, int B)
{
  const int w = h->w, npix = h->npix, L = h->L, nrec = h->c.nrec, hid = h->c.hidden, ns = h->nsub;
  const long rows = (long)B * npix, drows = (long)B * nrec * h->c.ny;
  int rc;
  if (fused_ok(h, x) && fused_decoder(h)) {
    if ((rc = decoder_bwd(h, B))) return rc;
    return layers_bwd_fused(h, x, B);
  }
  // decoder (pointwise MLP over the receivers' columns); drows is a multiple of ny
  if ((rc = splitk_grad(h, h->D1, hid, h->dpred, ns, drows, h->c.ny, h->grads + h->oW2))) return rc;
  if ((rc = colsum(h, h->dpred, drows, ns, 256, h->grads + h->oc2))) return rc;
  GEMM(h, mk(h->dpred, ns, 0, 0, h->W2b, ns, 0, 1, (int)drows, hid, ns, 1, h->dD1, hid, 0, 0));
  k_gelu_bwd<<<nblk(drows * hid), EW, 0, h->stream>>>(h->dD1, h->D1pre, h->dD1, drows * hid);
  if ((rc = splitk_grad(h, h->D0, w, h->dD1, hid, drows, h->c.ny, h->grads + h->oW1))) return rc;
  if ((rc = colsum(h, h->dD1, drows, hid, 256, h->grads + h->oc1))) return rc;
  GEMM(h, mk(h->dD1, hid, 0, 0, h->W1b, hid, 0, 1, (int)drows, w, hid, 1, h->dD0, w, 0, 0));
  if (fused_ok(h, x)) return layers_bwd_fused(h, x, B);
  if ((rc = need_wblk(h))) return rc;
  k_decoder_scatter<<<nblk(rows * w / 8), EW, 0, h->stream>>>(h->dD0, h->rec_x, B, nrec, h->c.ny, h->c.nx, w, h->dHa);
  // Fourier layers, last to first: dHa holds dL/dH[l+1]
  for (int l = L - 1; l >= 0; l--) {
    const bf16 *dA = h->dHa;
    if (l < L - 1) {
      k_gelu_bwd<<<nblk(rows * w), EW, 0, h->stream>>>(h->dHa, h->Apre[l], h->dA, rows * w);
      dA = h->dA;
    }
    if ((rc = weight_grad(h, h->H[l], w, dA, B, h->grads + h->oW[l]))) return rc;
    if ((rc = colsum(h, dA, rows, w, 1024, h->grads + h->ob[l]))) return rc;
    GEMM(h, mk(dA, w, 0, 0, h->Wb[l], w, 0, 1, (int)rows, w, w, 1, h->dHb, w, 0, 0));
    if ((rc = spectral_bwd(h, l, dA, B, h->dHb))) return rc;
    bf16 *t = h->dHa; h->dHa = h->dHb; h->dHb = t;
  }
  // lift
  if ((rc = weight_grad(h, x, h->c.cin, h->dHa, B, h->grads + h->oW0))) return rc;
  if ((rc = colsum(h, h->dHa, rows, w, 1024, h->grads + h->ob0))) return rc;
  NCK(h, cudaGetLastError());
  return 0;
}

}  // namespace

extern "C" const char *se2nn_last_error(const se2nn *h) { return h ? h->err : g_nn_create_err; }

extern "C" void se2nn_destroy(se2nn *h)
{
  if (!h) return;
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (void *p : h->allocs) cudaFree(p);
  delete h;
}

extern "C" long se2nn_num_params(const se2nn *h) { return h ? h->P : -1; }

extern "C" int se2nn_create(const se2nn_config *cfg, unsigned long long seed, se2nn **out)
{
  if (!out || !cfg) return nfail(nullptr, -1, "null argument");
  *out = nullptr;
  const se2nn_config c = *cfg;
  if (c.ny < 2 || c.nx < 2 || c.cin < 16 || c.cin % 16 || c.width < 16 || c.width % 16 || c.modes < 1 ||
      2 * c.modes > c.ny || 2 * c.modes > c.nx || c.layers < 1 || c.nrec < 1 || c.nout < c.ny || c.nout % c.ny ||
      c.hidden < 16 || c.hidden % 16 || c.max_batch < 1)
    return nfail(nullptr, -1, "invalid network configuration");
  if ((long)c.max_batch * c.ny > 65535 || 2L * c.modes * c.modes > 65535 ||
      ((long)c.max_batch * c.ny * c.nx + 63) / 64 > 65535)
    return nfail(nullptr, -1, "batch too large for the launch grid");
  se2nn *h = new se2nn();
  h->c = c;
  h->npix = c.ny * c.nx; h->w = c.width; h->m = c.modes; h->nmodes = 2 * c.modes * c.modes; h->L = c.layers;
  const int w = h->w, L = h->L, Bm = c.max_batch;
  const long nm = h->nmodes, npix = h->npix;
  // parameter layout
  long o = 0;
  h->oW0 = o; o += (long)c.cin * w;
  h->ob0 = o; o += w;
  for (int l = 0; l < L; l++) {
    h->oWre.push_back(o); o += nm * w * w;
    h->oWim.push_back(o); o += nm * w * w;
    h->oW.push_back(o); o += (long)w * w;
    h->ob.push_back(o); o += w;
  }
  h->nsub = c.nout / c.ny;
  h->oW1 = o; o += (long)w * c.hidden;
  h->oc1 = o; o += c.hidden;
  h->oW2 = o; o += (long)c.hidden * h->nsub;
  h->oc2 = o; o += h->nsub;
  h->P = o;
  h->split = (npix % 8 == 0) ? 8 : (npix % 4 == 0) ? 4 : (npix % 2 == 0) ? 2 : 1;
  int rc = 0;
#define TRY(x) do { if ((rc = (x)) != 0) { snprintf(g_nn_create_err, sizeof(g_nn_create_err), "%s", h->err); se2nn_destroy(h); return rc; } } while (0)
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    delete h;
    return nfail(nullptr, -2, "cudaStreamCreate failed");
  }
  {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      nfail(h, -2, "device query failed");
      TRY(-2);
    }
  }
  TRY(nalloc(h, &h->params, h->P));
  TRY(nalloc(h, &h->grads, h->P));
  TRY(nalloc(h, &h->adam_m, h->P));
  TRY(nalloc(h, &h->adam_v, h->P));
  TRY(nalloc(h, &h->Pb, h->P));
  h->W0b = h->Pb + h->oW0; h->W1b = h->Pb + h->oW1; h->W2b = h->Pb + h->oW2;
  for (int l = 0; l < L; l++) {
    h->Wb.push_back(h->Pb + h->oW[l]);
    h->Wreb.push_back(h->Pb + h->oWre[l]);
    h->Wimb.push_back(h->Pb + h->oWim[l]);
  }
  h->Wblk.assign(L, nullptr); h->Zp.assign(L, nullptr);
  h->H.assign(L + 1, nullptr); h->Apre.assign(L > 1 ? L - 1 : 0, nullptr);
  for (int l = 0; l < L; l++) {
    TRY(nalloc(h, &h->Wblk[l], (size_t)nm * 4 * w * w));
    TRY(nalloc(h, &h->Zp[l], (size_t)nm * Bm * 2 * w));
  }
  const size_t act = (size_t)Bm * npix * w;
  for (int l = 0; l <= L; l++) TRY(nalloc(h, &h->H[l], act));
  for (size_t l = 0; l < h->Apre.size(); l++) TRY(nalloc(h, &h->Apre[l], act));
  TRY(nalloc(h, &h->S, act));
  TRY(nalloc(h, &h->dHa, act));
  TRY(nalloc(h, &h->dHb, act));
  TRY(nalloc(h, &h->dA, act));
  TRY(nalloc(h, &h->Xf, (size_t)Bm * c.ny * 2 * h->m * w));
  TRY(nalloc(h, &h->Z, (size_t)Bm * 4 * h->m * h->m * w));
  TRY(nalloc(h, &h->Y, (size_t)Bm * 4 * h->m * h->m * w));
  TRY(nalloc(h, &h->Yy, (size_t)Bm * 2 * c.ny * h->m * w));
  TRY(nalloc(h, &h->Yp, (size_t)nm * Bm * 2 * w));
  TRY(nalloc(h, &h->dZp, (size_t)nm * Bm * 2 * w));
  const size_t drows = (size_t)Bm * c.nrec * c.ny;
  TRY(nalloc(h, &h->D0, drows * w));
  TRY(nalloc(h, &h->dD0, drows * w));
  TRY(nalloc(h, &h->D1pre, drows * c.hidden));
  TRY(nalloc(h, &h->D1, drows * c.hidden));
  TRY(nalloc(h, &h->dD1, drows * c.hidden));
  TRY(nalloc(h, &h->out, drows * h->nsub));
  TRY(nalloc(h, &h->dpred, drows * h->nsub));
  TRY(nalloc(h, &h->dblk, (size_t)nm * 4 * w * w));
  TRY(nalloc(h, &h->lpart, 1024));
  TRY(nalloc(h, &h->rec_x, (size_t)c.nrec));
  {
    const long wg = (long)Bm * h->split * (long)w * std::max(w, c.cin);
    const long cs1 = (((long)Bm * npix + 1023) / 1024) * w;
    const long cs2 = std::max((long)Bm * c.nrec * (long)c.hidden * std::max(w, h->nsub),
                              (((long)drows + 255) / 256) * std::max(h->nsub, c.hidden));
    h->partial_n = std::max(wg, std::max(cs1, cs2));
    // the partial sums, and those that only the fused kernels have beside them, in one allocation
    auto padded = [](size_t n) { return (n + 63) / 64 * 64; };
    const size_t np = padded((size_t)h->partial_n), nc = padded((size_t)cs1);
    const size_t nd = (size_t)Bm * c.nrec * c.hidden * h->nsub + (drows + 255) / 256 * (size_t)(h->nsub + c.hidden);
    TRY(nalloc(h, &h->partial, np + (fused_shape(h) ? nc + nd : 0)));
    h->colpart = h->partial + np;
    h->decpart = h->colpart + nc;
  }
  TRY(build_dft(h));
  TRY(fused_setup(h));
  // initial parameters (seeded)
  {
    std::vector<float> p(h->P, 0.f);
    uint64_t s = seed ^ 0x5EED5EED12345678ULL;
    for (long i = 0; i < (long)c.cin * w; i++) p[h->oW0 + i] = uniform_pm(&s, 1.0f / sqrtf((float)c.cin));
    for (int l = 0; l < L; l++) {
      for (long i = 0; i < nm * w * w; i++) p[h->oWre[l] + i] = uniform_pm(&s, 1.0f / (float)w);
      for (long i = 0; i < nm * w * w; i++) p[h->oWim[l] + i] = uniform_pm(&s, 1.0f / (float)w);
      for (long i = 0; i < (long)w * w; i++) p[h->oW[l] + i] = uniform_pm(&s, 1.0f / sqrtf((float)w));
    }
    for (long i = 0; i < (long)w * c.hidden; i++) p[h->oW1 + i] = uniform_pm(&s, 1.0f / sqrtf((float)w));
    for (long i = 0; i < (long)c.hidden * h->nsub; i++) p[h->oW2 + i] = uniform_pm(&s, 1.0f / sqrtf((float)c.hidden));
    if (cudaMemcpy(h->params, p.data(), h->P * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(h->grads, 0, h->P * 4) != cudaSuccess || cudaMemset(h->adam_m, 0, h->P * 4) != cudaSuccess ||
        cudaMemset(h->adam_v, 0, h->P * 4) != cudaSuccess) {
      nfail(h, -2, "parameter upload failed");
      TRY(-2);
    }
    std::vector<int> rx(c.nrec);
    for (int r = 0; r < c.nrec; r++) rx[r] = (int)(((2 * r + 1) * (long)c.nx) / (2 * c.nrec));
    if (cudaMemcpy(h->rec_x, rx.data(), c.nrec * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
      nfail(h, -2, "receiver upload failed");
      TRY(-2);
    }
  }
  TRY(refresh_bf16(h));
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) { nfail(h, -2, "set-up kernels failed"); TRY(-2); }
#undef TRY
  *out = h;
  return 0;
}

extern "C" int se2nn_set_stream(se2nn *h, void *stream)
{
  if (!h) return -1;
  NCK(h, cudaStreamSynchronize(h->stream));
  if (stream) h->stream = static_cast<cudaStream_t>(stream);
  return 0;
}

// Device -> the caller's host array.  Where its pages are not there yet, they are faulted in
// first by up to 16 host threads, one store each (the array is about to be overwritten): the copy
// alone faults them one after the other (us, copy alone -> this: 67 MB of new memory 3600 -> 2300, 9.5 MB 740 -> 590;
// into an array that is in use already nothing is touched: 363, 64.  A kernel that stored into the host
// array took 1230 and 133 there).
constexpr long TOUCH_BYTES = 4 << 20;   // per thread
static void touch_absent_pages(float *p, size_t bytes)
{
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = (uintptr_t)p / page * page;
  const long pages = (long)(((uintptr_t)p + bytes - a + page - 1) / page);
  int absent = 0;   // of three pages in it (asking for all of them takes 3 to 8 us)
  for (int k = 1; k < 6; k += 2) {
    unsigned char in = 0;
    if (mincore(reinterpret_cast<void *>(a + pages * k / 6 * page), page, &in) != 0) return;
    absent += !(in & 1);
  }
  if (absent < 2) return;
  auto touch = [=](long i0, long i1) {
    for (long i = i0; i < i1; i++) *reinterpret_cast<volatile char *>(std::max(a + i * page, (uintptr_t)p)) = 0;
  };
  const long nt = std::max(1L, std::min((long)std::min(16u, std::thread::hardware_concurrency()), (long)bytes / TOUCH_BYTES));
  std::thread th[16];
  for (long t = 1; t < nt; t++) {
    try {
      th[t] = std::thread(touch, pages * t / nt, pages * (t + 1) / nt);
    } catch (...) {   // (no more threads: this one does the part)
      touch(pages * t / nt, pages * (t + 1) / nt);
    }
  }
  touch(0, pages / nt);
  for (std::thread &t : th)
    if (t.joinable()) t.join();
}

static int copy_out(se2nn *h, float *dst, const float *src, long n)
{
  NCK(h, cudaStreamSynchronize(h->stream));   // (earlier work may still read the array)
  const size_t bytes = (size_t)n * sizeof(float);
  if (bytes >= 2 * TOUCH_BYTES) {   // (one thread gains nothing, and asking takes 2 of the 13 us of a small copy)
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) cudaGetLastError();
    else if (at.type != cudaMemoryTypeDevice) touch_absent_pages(dst, bytes);   // (the host cannot store there)
  }
  NCK(h, cudaMemcpy(dst, src, n * 4, cudaMemcpyDeviceToHost));
  return 0;
}

extern "C" int se2nn_get_params(se2nn *h, float *p)
{
  if (!h || !p) return -1;
  return copy_out(h, p, h->params, h->P);
}

extern "C" int se2nn_set_params(se2nn *h, const float *p)
{
  if (!h || !p) return -1;
  NCK(h, cudaStreamSynchronize(h->stream));
  NCK(h, cudaMemcpy(h->params, p, h->P * 4, cudaMemcpyHostToDevice));
  int rc = refresh_bf16(h);
  if (rc) return rc;
  NCK(h, cudaStreamSynchronize(h->stream));
  return 0;
}

extern "C" int se2nn_get_grads(se2nn *h, float *g)
{
  if (!h || !g) return -1;
  return copy_out(h, g, h->grads, h->P);
}

extern "C" int se2nn_set_receivers(se2nn *h, const int *rec_x)
{
  if (!h || !rec_x) return -1;
  for (int r = 0; r < h->c.nrec; r++)
    if (rec_x[r] < 0 || rec_x[r] >= h->c.nx) return nfail(h, -1, "receiver %d: cell %d outside 0..%d", r, rec_x[r], h->c.nx - 1);
  NCK(h, cudaStreamSynchronize(h->stream));
  NCK(h, cudaMemcpy(h->rec_x, rec_x, h->c.nrec * 4, cudaMemcpyHostToDevice));
  return 0;
}

static int check_batch(se2nn *h, int batch)
{
  if (batch < 1 || batch > h->c.max_batch) return nfail(h, -1, "batch %d outside 1..%d", batch, h->c.max_batch);
  return 0;
}

extern "C" int se2nn_forward(se2nn *h, const void *x_dev, int batch, float *out_dev)
{
  if (!h || !x_dev || !out_dev) return -1;
  int rc = check_batch(h, batch);
  if (rc) return rc;
  return forward(h, static_cast<const bf16 *>(x_dev), batch, out_dev, false);
}

extern "C" int se2nn_loss_grad(se2nn *h, const void *x_dev, int batch, const float *target_dev, double *loss,
                               float *out_dev)
{
  if (!h || !x_dev || !target_dev) return -1;
  int rc = check_batch(h, batch);
  if (rc) return rc;
  const bf16 *x = static_cast<const bf16 *>(x_dev);
  float *out = out_dev ? out_dev : h->out;
  if ((rc = forward(h, x, batch, out, true))) return rc;
  const long n = (long)batch * h->c.nrec * h->c.nout;
  const int nb = (int)std::min<long>(1024, (n + EW - 1) / EW);
  k_mse<<<nb, EW, 0, h->stream>>>(out, target_dev, n, h->lpart, h->dpred);
  NCK(h, cudaGetLastError());
  if ((rc = backward(h, x, batch))) return rc;
  std::vector<double> part(nb);
  NCK(h, cudaMemcpyAsync(part.data(), h->lpart, nb * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  NCK(h, cudaStreamSynchronize(h->stream));
  double s = 0.0;
  for (int i = 0; i < nb; i++) s += part[i];
  if (loss) *loss = s / (double)n;
  return 0;
}

extern "C" int se2nn_adam_step(se2nn *h, float lr, float beta1, float beta2, float eps, float weight_decay)
{
  if (!h) return -1;
  h->adam_t++;
  const float c1 = 1.f - powf(beta1, (float)h->adam_t), c2 = 1.f - powf(beta2, (float)h->adam_t);
  k_adam<<<nblk((h->P + 3) / 4), EW, 0, h->stream>>>(h->params, h->grads, h->adam_m, h->adam_v, h->Pb, h->P, lr, beta1, beta2, eps,
                                            weight_decay, c1, c2);
  NCK(h, cudaGetLastError());
  return params_changed(h);
}

extern "C" int se2nn_build_inputs(se2nn *h, const void *materials_dev, const float *src_dev, const int *idx_dev,
                                  int batch, float sigma_cells, void *x_dev)
{
  if (!h || !materials_dev || !src_dev || !idx_dev || !x_dev || !(sigma_cells > 0.f)) return -1;
  int rc = check_batch(h, batch);
  if (rc) return rc;
  k_build_inputs<<<nblk((long)batch * h->npix), EW, 0, h->stream>>>(
      static_cast<const float *>(materials_dev), src_dev, idx_dev, batch, h->c.ny, h->c.nx, h->c.cin,
      1.0f / (2.0f * sigma_cells * sigma_cells), static_cast<bf16 *>(x_dev));
  NCK(h, cudaGetLastError());
  return 0;
}

extern "C" int se2nn_gather_targets(se2nn *h, const float *targets_dev, const int *idx_dev, int batch, float *out_dev)
{
  if (!h || !targets_dev || !idx_dev || !out_dev) return -1;
  int rc = check_batch(h, batch);
  if (rc) return rc;
  const long row = (long)h->c.nrec * h->c.nout;
  k_gather_rows<<<nblk(batch * row), EW, 0, h->stream>>>(targets_dev, idx_dev, batch, row, out_dev);
  NCK(h, cudaGetLastError());
  return 0;
}

extern "C" int se2nn_set_tensor_path(int mode)
{
  if (mode < 0 || mode > 2) return -1;
  g_tc_path = mode;
  return 0;
}

extern "C" int se2nn_tensor_path_info(long out[3])
{
  if (!out) return -1;
  int flag = 0;   // (the current device's flag)
  if (cudaMemcpyFromSymbol(&flag, g_tc_err, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  out[0] = g_tc_launches.load();
  out[1] = g_mma_launches.load();
  out[2] = flag;
  return 0;
}

extern "C" int se2nn_gemm(const void *A_dev, const void *B_dev, float *C_dev, int M, int N, int K, int batch, long lda,
                          long ldb, long ldc, long sA, long sB, long sC, int transA, int transB, float alpha, float beta,
                          void *stream)
{
  if (!A_dev || !B_dev || !C_dev || M < 1 || N < 1 || K < 1 || batch < 1) return nfail(nullptr, -1, "bad GEMM arguments");
  GemmArgs g = mk(static_cast<const bf16 *>(A_dev), lda, sA, transA, static_cast<const bf16 *>(B_dev), ldb, sB, transB,
                  M, N, K, batch, C_dev, ldc, sC, 1);
  g.alpha = alpha;
  g.beta = beta;
  if (beta != 0.f) { g.Cin = C_dev; g.ldcin = ldc; g.sCin = sC; g.cin_f32 = 1; }
  cudaError_t e = launch_gemm(g, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return nfail(nullptr, -2, "GEMM launch: %s", cudaGetErrorString(e));
  return 0;
}
