// Memory-bound helper kernels of the learned preconditioner (layouts,
// pooling, upsampling, the 2-channel input and 1-channel output
// convolutions, weight packing, optimiser, loss): plain SIMT code.  The
// heavy 3x3 convolutions run on the tensor cores (nn_gemm.cu).
//
// Activations are bf16 NHWC; a tensor may be a channel slice [coff, coff+c)
// of a wider one with cstride channels per pixel.  Channel counts, strides
// and offsets are multiples of 8 (16-byte channel vectors).
#include <cuda_bf16.h>
#include <stdint.h>

#include "sgb_common.cuh"

namespace sgb {
namespace nn {
namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float ld(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ bf16 st(float v) { return __float2bfloat16_rn(v); }

int blocks_for(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b > 152 * 32 ? 152 * 32 : (b < 1 ? 1 : b));
}

// 8 bf16 channels moved as one 16-byte vector (little-endian pairs: the
// lower half of each 32-bit word is the even channel).
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f[2 * k] = __uint_as_float(w[k] << 16);
    f[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  unsigned w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    w[k] = *reinterpret_cast<const unsigned*>(&h2);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// Plain loads: the tensors may be what the launch before this one writes, and
// that launch may still be running when this grid starts (see pdl_wait).
__device__ __forceinline__ uint4 ld8(const bf16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st8(bf16* p, const uint4& v) { *reinterpret_cast<uint4*>(p) = v; }

// Every kernel here is a programmatic dependent of the launch before it (pdl_wait
// at its start): a prediction is some 16 launches of 4 - 30 us.
template <class... P, class... A>
void launch_nn(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
  launch_pdl(kern, grid, block, smem, s, args...);  // a failure stays for cudaGetLastError
}

#define GRID_STRIDE(i, total) \
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (total); i += (long long)gridDim.x * blockDim.x)

// out[k][n][c][y][x] = in[n][y][x - 1 + k][coff + c] (one copy: k = 1).
// A block moves a tile of 32 columns (plus the one-column halo the shifted
// copies read) of one image row through shared memory: 16-byte reads of
// the channel vectors, 64-byte coalesced rows of the channel-major output.
constexpr int TCHW_X = 32;
__global__ void to_chw_kernel(int n, int h, int w, int c, int cstride, int coff, const bf16* in, int copies,
                              bf16* out) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) bf16 tile[];  // [TCHW_X + 2][c]
  const int row = blockIdx.y;  // b * h + y
  const int x0 = blockIdx.x * TCHW_X;
  const int cv = c / 8;
  for (int q = threadIdx.x; q < (TCHW_X + 2) * cv; q += blockDim.x) {
    const int px = q / cv, k8 = (q % cv) * 8;
    const int x = x0 - 1 + px;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (x >= 0 && x < w) v = ld8(in + ((long long)row * w + x) * cstride + coff + k8);
    st8(tile + px * c + k8, v);
  }
  __syncthreads();
  const long long plane = (long long)n * c * h * w;
  const int b = row / h, y = row % h;
  for (int q = threadIdx.x; q < copies * c * TCHW_X; q += blockDim.x) {
    const int xx = q % TCHW_X;
    const int ch = (q / TCHW_X) % c;
    const int k = q / (TCHW_X * c);
    const int x = x0 + xx;
    if (x >= w) continue;
    const int shift = copies == 1 ? 0 : k - 1;
    out[k * plane + (((long long)b * c + ch) * h + y) * w + x] = tile[(xx + 1 + shift) * c + ch];
  }
}

// Input convolution: 2 fp32 channels [n][2][h][w] -> c bf16 channels (ReLU).
// A thread computes CIN_PX adjacent pixels of a row, so that a weight read from
// shared memory (where it fits, as a broadcast of the whole block) serves that
// many multiply-adds; with one pixel per thread the kernel was bound by those
// reads (53 us for 32 channels of 8 x 256 x 512 pixels).
constexpr int CIN_PX = 4;
template <bool SMEM_W>
__global__ void __launch_bounds__(128) conv_in_fwd_kernel(int n, int h, int w, int c, const float* in, const float* W,
                                                          const float* b, bf16* out, int cstride, int coff) {
  pdl_wait();
  pdl_trigger();
  // weights of 8 output channels side by side: [c / 8][18 taps + bias][8]
  extern __shared__ __align__(16) float cin_w[];
  if (SMEM_W) {
    for (int k = threadIdx.x; k < 19 * c; k += blockDim.x) {
      const int co = k / 19, t = k - 19 * co;
      cin_w[(co / 8 * 19 + t) * 8 + co % 8] = t < 18 ? W[co * 18 + t] : b[co];
    }
    __syncthreads();
  }
  const int wq = (w + CIN_PX - 1) / CIN_PX;
  const long long total = (long long)n * h * wq;
  GRID_STRIDE(i, total) {
    const int x = (int)(i % wq) * CIN_PX;
    const int y = (int)((i / wq) % h);
    const int bb = (int)(i / ((long long)wq * h));
    float v[6][CIN_PX + 2];  // [channel, ky][x - 1 ..]
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const int yy = y - 1 + r % 3;
      const float* p = in + (((long long)bb * 2 + r / 3) * h + yy) * w;
#pragma unroll
      for (int k = 0; k < CIN_PX + 2; ++k) {
        const int xx = x - 1 + k;
        v[r][k] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? p[xx] : 0.f;
      }
    }
    bf16* o = out + (((long long)bb * h + y) * w + x) * cstride + coff;
    for (int c8 = 0; c8 < c; c8 += 8) {
      float a[CIN_PX][8];
#pragma unroll
      for (int t = -1; t < 18; ++t) {  // the bias, then the taps
        float wt[8];
        if (SMEM_W) {
          const float4* q = reinterpret_cast<const float4*>(cin_w + (c8 / 8 * 19 + (t < 0 ? 18 : t)) * 8);
          const float4 q0 = q[0], q1 = q[1];
          wt[0] = q0.x; wt[1] = q0.y; wt[2] = q0.z; wt[3] = q0.w;
          wt[4] = q1.x; wt[5] = q1.y; wt[6] = q1.z; wt[7] = q1.w;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) wt[j] = t < 0 ? b[c8 + j] : W[(c8 + j) * 18 + t];  // plain loads, see ld8
        }
#pragma unroll
        for (int k = 0; k < CIN_PX; ++k)
#pragma unroll
          for (int j = 0; j < 8; ++j) a[k][j] = t < 0 ? wt[j] : fmaf(wt[j], v[(t < 0 ? 0 : t) / 3][k + (t < 0 ? 0 : t) % 3], a[k][j]);
      }
#pragma unroll
      for (int k = 0; k < CIN_PX; ++k) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[k][j] = a[k][j] > 0.f ? a[k][j] : 0.f;
        if (x + k < w) st8(o + (long long)k * cstride + c8, pack8(a[k]));
      }
    }
  }
}

// Output convolution: c bf16 channels -> 1 fp32 channel (linear).
__global__ void conv_out_fwd_kernel(int n, int h, int w, int c, const bf16* in, int cstride, const float* W,
                                    const float* b, float* out) {
  pdl_wait();
  pdl_trigger();
  const long long total = (long long)n * h * w;
  GRID_STRIDE(i, total) {
    const int x = (int)(i % w);
    const int y = (int)((i / w) % h);
    const int bb = (int)(i / ((long long)w * h));
    float a = b[0];
    for (int ky = 0; ky < 3; ++ky)
      for (int kx = 0; kx < 3; ++kx) {
        const int yy = y - 1 + ky, xx = x - 1 + kx;
        if (yy < 0 || yy >= h || xx < 0 || xx >= w) continue;
        const bf16* p = in + (((long long)bb * h + yy) * w + xx) * cstride;
        for (int c8 = 0; c8 < c; c8 += 8) {
          float f[8];
          unpack8(ld8(p + c8), f);
#pragma unroll
          for (int j = 0; j < 8; ++j) a = fmaf(W[(c8 + j) * 9 + ky * 3 + kx], f[j], a);
        }
      }
    out[i] = a;
  }
}

// The same convolution for 32 or 64 channels from shared memory: a block of
// COUT_TX threads takes COUT_TX columns of COUT_R rows, stages the COUT_R + 2
// input rows (with the column halo, c channels, 16-byte vectors) and the
// weights (tap-major) once, and each thread sums its column's COUT_R pixels,
// each weight read serving all of them.  A thread walks a pixel's channel
// vectors starting at (lane mod c/8), so that the 8 threads of a 16-byte access
// phase hit distinct banks.  One row per block staged every row three times
// and read the weights once per pixel: 80 us for 32 channels of 8 x 256 x 512.
constexpr int COUT_TX = 128, COUT_R = 4;
template <int CV>  // channel vectors per pixel (c = 8 CV)
__global__ void __launch_bounds__(COUT_TX) conv_out_tile_kernel(int n, int h, int w, const bf16* in, int cstride,
                                                                 const float* W, const float* b, float* out) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char cout_smem[];
  constexpr int cv = CV, c = 8 * CV, cols = COUT_TX + 2, rows = COUT_R + 2;
  uint4* srow = reinterpret_cast<uint4*>(cout_smem);  // [rows][cols][cv]
  float* ws = reinterpret_cast<float*>(srow + rows * cols * cv);  // [9][c]
  const int ntx = (w + COUT_TX - 1) / COUT_TX, nty = (h + COUT_R - 1) / COUT_R;
  const int x0 = (blockIdx.x % ntx) * COUT_TX;
  const int y0 = (blockIdx.x / ntx % nty) * COUT_R, bb = blockIdx.x / (ntx * nty);
  for (int k = threadIdx.x; k < 9 * c; k += COUT_TX) {
    const int tap = k / c, ci = k - tap * c;
    ws[k] = W[ci * 9 + tap];
  }
  // eight vectors per thread in flight at a time: loads first, then stores
  constexpr int nvec = rows * cols * cv;
  for (int k0 = threadIdx.x; k0 < nvec; k0 += 8 * COUT_TX) {
    uint4 q[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * COUT_TX;
      q[u] = make_uint4(0u, 0u, 0u, 0u);
      if (k < nvec) {
        const int v = k % cv, rc = k / cv;
        const int col = rc % cols, r = rc / cols;
        const int yy = y0 - 1 + r, xx = x0 - 1 + col;
        if (yy >= 0 && yy < h && xx >= 0 && xx < w) q[u] = ld8(in + (((long long)bb * h + yy) * w + xx) * cstride + 8 * v);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k0 + u * COUT_TX < nvec) srow[k0 + u * COUT_TX] = q[u];
  }
  __syncthreads();
  const int t = threadIdx.x, x = x0 + t;
  if (x >= w) return;
  float acc[COUT_R][4];  // four partial sums per pixel: short FMA chains
#pragma unroll
  for (int i = 0; i < COUT_R; ++i) {
    acc[i][0] = b[0];
    acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  }
#pragma unroll 3
  for (int tap = 0; tap < 9; ++tap) {
    const int ky = tap / 3, kx = tap - 3 * ky;
    const uint4* px = srow + (ky * cols + t + kx) * cv;
    const float* wt = ws + tap * c;
#pragma unroll
    for (int vv = 0; vv < cv; ++vv) {
      const int v = (vv + t) & (cv - 1);
      const float4 w0 = lds4(wt + 8 * v), w1 = lds4(wt + 8 * v + 4);
      const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < COUT_R; ++i) {
        float f[8];
        unpack8(px[i * cols * cv + v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j & 3] = fmaf(wv[j], f[j], acc[i][j & 3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < COUT_R; ++i)
    if (y0 + i < h) out[((long long)bb * h + y0 + i) * w + x] = (acc[i][0] + acc[i][1]) + (acc[i][2] + acc[i][3]);
}

// Data gradient of the output convolution, times [act > 0] (the ReLU of the
// layer that produced its input): dx[p][ci] = sum_tap W[ci][tap] g[p - off].
// A thread takes one channel vector of COD_PX adjacent pixels of a row, so that
// the 72 weights it reads (shared memory, tap-major) serve all of them; with
// the weights read from global memory for every pixel it took 60 us for 32
// channels of 8 x 256 x 512.
constexpr int COD_PX = 4;
__global__ void __launch_bounds__(256) conv_out_dgrad_kernel(int n, int h, int w, int c, const float* g, const float* W,
                                                             const bf16* act, int act_cstride, bf16* dx) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) float cod_w[];  // [9][c]
  for (int k = threadIdx.x; k < 9 * c; k += blockDim.x) cod_w[k] = W[(k % c) * 9 + k / c];
  __syncthreads();
  const int cv = c / 8, wq = (w + COD_PX - 1) / COD_PX;
  const long long total = (long long)n * h * wq * cv;
  GRID_STRIDE(i, total) {
    const int c8 = (int)(i % cv) * 8;
    const long long q = i / cv;
    const int x = (int)(q % wq) * COD_PX;
    const int y = (int)((q / wq) % h);
    const int bb = (int)(q / ((long long)wq * h));
    float gv[3][COD_PX + 2];  // rows y + 1, y, y - 1; columns x - 1 ..
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int yy = y + 1 - r;
      const float* p = g + ((long long)bb * h + yy) * w;
#pragma unroll
      for (int k = 0; k < COD_PX + 2; ++k) {
        const int xx = x - 1 + k;
        gv[r][k] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? p[xx] : 0.f;
      }
    }
    float o[COD_PX][8];
#pragma unroll
    for (int k = 0; k < COD_PX; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) o[k][j] = 0.f;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      // output pixel (y + 1 - ky, x + 1 - kx) reads this pixel through tap (ky, kx)
      const float4 w0 = lds4(cod_w + t * c + c8), w1 = lds4(cod_w + t * c + c8 + 4);
      const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int k = 0; k < COD_PX; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) o[k][j] = fmaf(wv[j], gv[t / 3][k + 2 - t % 3], o[k][j]);
    }
    const long long pix = ((long long)bb * h + y) * w + x;
#pragma unroll
    for (int k = 0; k < COD_PX; ++k) {
      if (x + k >= w) break;
      float m[8];
      unpack8(ld8(act + (pix + k) * act_cstride + c8), m);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[k][j] = m[j] > 0.f ? o[k][j] : 0.f;
      st8(dx + (pix + k) * c + c8, pack8(o[k]));
    }
  }
}

// Weight and bias gradients of the input and output convolutions:
//   dW[c][k] += sum_p v[p][c] s[p + d_k],  d_k the nine taps' offsets,
// v a bf16 NHWC tensor (channel vectors of 8), s an fp32 image (0 outside).
// Input convolution: v = dy, s = an input channel, d_k = (ky - 1, kx - 1);
// output convolution: v = the layer's input, s = dy, d_k = (1 - ky, 1 - kx).
// A thread owns one column and VS_C = 8 / NI channels, walks VS_ROWS rows with
// the 3 x 3 windows of the NI images in registers and keeps the 72 sums of its
// channels; each v vector is read once.  One block per channel with scalar reads
// at the pixel stride took 553 us (output) and 398 us (input) for 32 channels of
// 8 x 256 x 512 pixels; 16 rows per block, whose 80 sums per thread then meet
// through shuffles, 99 us (output) and 2 x 74 us (input, one image at a time).
constexpr int VS_ROWS = 64, VS_X = 64;  // rows and columns per block
template <int SIGN, int NI, bool VEC>
__global__ void __launch_bounds__(256) vec_scalar_wgrad_kernel(int h, int w, int c, const bf16* v, int v_cstride,
                                                               const float* s, float* dW, float* db_vec,
                                                               float* db_scalar) {
  pdl_wait();
  pdl_trigger();
  constexpr int VS_C = 8 / NI, CG = 256 / VS_X;  // channels per thread, channel groups per block
  // the block's part of the images with its halo (0 outside); then the warps' sums
  constexpr int TW = VS_X + 2, TILE = NI * (VS_ROWS + 2) * TW, RED = 8 * CG * (9 * NI + 1) * VS_C;
  __shared__ float sm[TILE > RED ? TILE : RED];
  const int cg = threadIdx.x % CG, c0 = (blockIdx.y * CG + cg) * VS_C;
  const int ntx = (w + VS_X - 1) / VS_X, nty = (h + VS_ROWS - 1) / VS_ROWS;
  const int x = (blockIdx.x % ntx) * VS_X + threadIdx.x / CG;
  const int y0 = (blockIdx.x / ntx % nty) * VS_ROWS, n = blockIdx.x / (ntx * nty);
  const bool in = x < w && c0 < c;
  const long long hw = (long long)h * w;
  const float* img = s + n * NI * hw;
  const bf16* vp = v + ((long long)n * h + y0) * w * v_cstride + (long long)x * v_cstride + c0;
  float acc[NI][9][VS_C], bias[VS_C], sc = 0.f;
  auto vec = [&](int r, float (&f)[VS_C]) {  // 0 beyond the image or the channels
    const bf16* q = vp + (long long)r * w * v_cstride;
    const bool ok = in && y0 + r < h;
    if constexpr (!VEC) {
#pragma unroll
      for (int j = 0; j < VS_C; ++j) f[j] = ok && c0 + j < c ? ld(q + j) : 0.f;
    } else if constexpr (VS_C == 8) {
      unpack8(ok ? ld8(q) : make_uint4(0u, 0u, 0u, 0u), f);
    } else {
      const uint2 u = ok ? *reinterpret_cast<const uint2*>(q) : make_uint2(0u, 0u);
      f[0] = __uint_as_float(u.x << 16);
      f[1] = __uint_as_float(u.x & 0xffff0000u);
      f[2] = __uint_as_float(u.y << 16);
      f[3] = __uint_as_float(u.y & 0xffff0000u);
    }
  };
#pragma unroll
  for (int j = 0; j < VS_C; ++j) {
    bias[j] = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int k = 0; k < 9; ++k) acc[i][k][j] = 0.f;
  }
  float zero = 0.f;  // NaN after an infinity or NaN of the image
  for (int q = threadIdx.x; q < TILE; q += 256) {
    const int i = q / ((VS_ROWS + 2) * TW), rr = q / TW % (VS_ROWS + 2), cc = q % TW;
    const int yy = y0 - 1 + rr, xx = blockIdx.x % ntx * VS_X - 1 + cc;
    const float u = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? img[i * hw + (long long)yy * w + xx] : 0.f;
    sm[q] = u;
    zero = fmaf(u, 0.f, zero);
  }
  __syncthreads();
  const float* tile = sm + threadIdx.x / CG;
  // four rows' vector loads are issued together
#pragma unroll 1
  for (int r0 = 0; r0 < VS_ROWS && y0 + r0 < h; r0 += 4) {
    float f[4][VS_C], win[NI][6][3];
#pragma unroll
    for (int r = 0; r < 4; ++r) vec(r0 + r, f[r]);
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) win[i][q][d] = tile[(i * (VS_ROWS + 2) + r0 + q) * TW + d];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (in && y0 + r0 + r < h) sc += win[0][r + 1][1];
#pragma unroll
      for (int j = 0; j < VS_C; ++j) {
        bias[j] += f[r][j];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
          for (int k = 0; k < 9; ++k) {
            const int t = SIGN > 0 ? k : 8 - k;
            acc[i][k][j] = fmaf(f[r][j], win[i][r + t / 3][t % 3], acc[i][k][j]);
          }
      }
    }
  }
  // The loop above also multiplies what takes no part: pixels beyond the images, and
  // for the input convolution zero gradients.  That adds 0 where all is finite; else
  // (a sum of v, or `zero`, shows it) the sums are taken again without.
  bool redo = !(zero == 0.f);
#pragma unroll
  for (int j = 0; j < VS_C; ++j) redo |= !(bias[j] - bias[j] == 0.f);
  if (__syncthreads_or(redo)) {
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int k = 0; k < 9; ++k)
#pragma unroll
        for (int j = 0; j < VS_C; ++j) acc[i][k][j] = 0.f;
#pragma unroll 1
    for (int r = 0; r < VS_ROWS && y0 + r < h; ++r) {
      float f[VS_C];
      vec(r, f);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int t = SIGN > 0 ? k : 8 - k, yy = y0 + r - 1 + t / 3, xx = x - 1 + t % 3;
        if (!in || yy < 0 || yy >= h || xx < 0 || xx >= w) continue;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const float u = tile[(i * (VS_ROWS + 2) + r + t / 3) * TW + t % 3];
#pragma unroll
          for (int j = 0; j < VS_C; ++j)
            if (SIGN < 0 || f[j] != 0.f) acc[i][k][j] = fmaf(f[j], u, acc[i][k][j]);
        }
      }
    }
  }
  // lanes of equal cg, then the block's warps, then one addition per sum
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  auto red = [&](int u, int g, int k, int j) -> float& { return sm[((u * CG + g) * (9 * NI + 1) + k) * VS_C + j]; };
#pragma unroll
  for (int k = 0; k <= 9 * NI; ++k)
#pragma unroll
    for (int j = 0; j < VS_C; ++j) {
      float a = k < 9 * NI ? acc[k / 9 < NI ? k / 9 : 0][k % 9][j] : bias[j];
#pragma unroll
      for (int o = 16; o >= CG; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane < CG) red(wid, lane, k, j) = a;
    }
  __syncthreads();
  for (int q = threadIdx.x; q < CG * (9 * NI + 1) * VS_C; q += 256) {
    const int j = q % VS_C, k = q / VS_C % (9 * NI + 1), g = q / (VS_C * (9 * NI + 1));
    const int ch = (blockIdx.y * CG + g) * VS_C + j;
    float a = 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u) a += red(u, g, k, j);
    if (ch < c) {
      if (k < 9 * NI)
        atomicAdd(dW + (long long)ch * 9 * NI + k, a);
      else if (db_vec != nullptr)
        atomicAdd(db_vec + ch, a);
    }
  }
  if (db_scalar != nullptr && blockIdx.y == 0) {
    if (cg != 0) sc = 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sc += __shfl_xor_sync(0xffffffffu, sc, o);
    if (lane == 0) atomicAdd(db_scalar, sc);
  }
}

// 2x2 average pooling; h, w are the input dims; 8 channels per thread.
__global__ void pool2_kernel(int n, int h, int w, int c, const bf16* in, int cs_in, int coff_in, bf16* out) {
  pdl_wait();
  pdl_trigger();
  const int ho = h / 2, wo = w / 2, cv = c / 8;
  const long long total = (long long)n * ho * wo * cv;
  GRID_STRIDE(i, total) {
    const int c8 = (int)(i % cv) * 8;
    long long r = i / cv;
    const int x = (int)(r % wo);
    r /= wo;
    const int y = (int)(r % ho);
    const int b = (int)(r / ho);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int dy = 0; dy < 2; ++dy)
      for (int dx = 0; dx < 2; ++dx) {
        float f[8];
        unpack8(ld8(in + (((long long)b * h + 2 * y + dy) * w + 2 * x + dx) * cs_in + coff_in + c8), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += f[j];
      }
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= 0.25f;
    st8(out + (((long long)b * ho + y) * wo + x) * c + c8, pack8(acc));
  }
}

// Nearest 2x upsampling into a channel slice; h, w are the output dims;
// 8 channels per thread.
__global__ void up2_kernel(int n, int h, int w, int c, const bf16* in, bf16* out, int cs_out, int coff_out) {
  pdl_wait();
  pdl_trigger();
  const int cv = c / 8;
  const long long total = (long long)n * h * w * cv;
  GRID_STRIDE(i, total) {
    const int c8 = (int)(i % cv) * 8;
    long long r = i / cv;
    const int x = (int)(r % w);
    r /= w;
    const int y = (int)(r % h);
    const int b = (int)(r / h);
    st8(out + (((long long)b * h + y) * w + x) * cs_out + coff_out + c8,
        ld8(in + (((long long)b * (h / 2) + y / 2) * (w / 2) + x / 2) * c + c8));
  }
}

// 8 fp32 values of an fp32 gradient (two 16-byte loads).
__device__ __forceinline__ void ld8f(const float* p, float (&f)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// Gradient through the upsampling (sum of the 2x2 children of a channel
// slice of g, fp32) times [act > 0]; h, w are the fine dims; 8 channels per
// thread.
__global__ void up2_bwd_kernel(int n, int h, int w, int c, const float* g, int cs_g, int coff_g, const bf16* act,
                               bf16* out) {
  pdl_wait();
  pdl_trigger();
  const int ho = h / 2, wo = w / 2, cv = c / 8;
  const long long total = (long long)n * ho * wo * cv;
  GRID_STRIDE(i, total) {
    const int c8 = (int)(i % cv) * 8;
    long long r = i / cv;
    const int x = (int)(r % wo);
    r /= wo;
    const int y = (int)(r % ho);
    const int b = (int)(r / ho);
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int dy = 0; dy < 2; ++dy)
      for (int dx = 0; dx < 2; ++dx) {
        float f[8];
        ld8f(g + (((long long)b * h + 2 * y + dy) * w + 2 * x + dx) * cs_g + coff_g + c8, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += f[j];
      }
    const long long o = (((long long)b * ho + y) * wo + x) * c + c8;
    float m[8];
    unpack8(ld8(act + o), m);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = m[j] > 0.f ? a[j] : 0.f;
    st8(out + o, pack8(a));
  }
}

// Gradient at an encoder output: pooling backward (gp / 4 from the coarse
// level) plus the skip branch (a channel slice of g), times [act > 0];
// h, w are the fine dims; 8 channels per thread.
__global__ void pool2_bwd_kernel(int n, int h, int w, int c, const float* gp, const float* gs, int cs_s, int coff_s,
                                 const bf16* act, int cs_a, int coff_a, bf16* out) {
  pdl_wait();
  pdl_trigger();
  const int cv = c / 8;
  const long long total = (long long)n * h * w * cv;
  GRID_STRIDE(i, total) {
    const int c8 = (int)(i % cv) * 8;
    long long r = i / cv;
    const int x = (int)(r % w);
    r /= w;
    const int y = (int)(r % h);
    const int b = (int)(r / h);
    const long long pix = ((long long)b * h + y) * w + x;
    float a[8], f[8], m[8];
    ld8f(gp + (((long long)b * (h / 2) + y / 2) * (w / 2) + x / 2) * c + c8, a);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] *= 0.25f;
    if (gs != nullptr) {
      ld8f(gs + pix * cs_s + coff_s + c8, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += f[j];
    }
    unpack8(ld8(act + pix * cs_a + coff_a + c8), m);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = m[j] > 0.f ? a[j] : 0.f;
    st8(out + pix * c + c8, pack8(a));
  }
}

// db[c] += sum over images and pixels of dy[n][c][p] (channel-major copy);
// block (split, channel).
__global__ void bias_grad_kernel(int n, long long hw, int c, const bf16* dy, float* db) {
  pdl_wait();
  pdl_trigger();
  const int ch = blockIdx.y;
  float a = 0.f;
  const long long total = (long long)n * hw;
  GRID_STRIDE(q, total) {
    const long long b = q / hw, p = q % hw;
    a += ld(dy + (b * c + ch) * hw + p);
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(db + ch, a);
}

// db[c] += sum over pixels of dy[pixel][c] (NHWC): a thread sums 8 channels of
// every blockDim / (c / 8)-th pixel of its block's range, the block's threads of
// one vector meet in shared memory.
__global__ void __launch_bounds__(256) bias_grad_nhwc_kernel(long long pixels, int c, const bf16* dy, float* db) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ float bsum[];  // [c]
  const int cv = c / 8, per = 256 / cv, v = threadIdx.x % cv, p0 = threadIdx.x / cv;
  for (int k = threadIdx.x; k < c; k += 256) bsum[k] = 0.f;
  __syncthreads();
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (p0 < per) {
#pragma unroll 8
    for (long long p = (long long)blockIdx.x * per + p0; p < pixels; p += (long long)gridDim.x * per) {
      float f[8];
      unpack8(ld8(dy + p * c + 8 * v), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += f[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) atomicAdd(bsum + 8 * v + j, a[j]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < c; k += 256) atomicAdd(db + k, bsum[k]);
}

// fp32 [cout][cin][3][3] -> bf16 [cout][9][cin] and flipped transpose [cin][9][cout].
__global__ void pack_weights_kernel(int cout, int cin, const float* W, bf16* wt, bf16* wflip) {
  pdl_wait();
  pdl_trigger();
  const long long total = (long long)cout * cin * 9;
  GRID_STRIDE(i, total) {
    const int t = (int)(i % 9);
    const int ci = (int)((i / 9) % cin);
    const int co = (int)(i / (9LL * cin));
    const bf16 v = st(W[i]);
    wt[((long long)co * 9 + t) * cin + ci] = v;
    if (wflip != nullptr) wflip[((long long)ci * 9 + (8 - t)) * cout + co] = v;
  }
}

__global__ void adam_kernel(long long n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                            float eps, float c1, float c2, float wd) {
  pdl_wait();
  pdl_trigger();
  GRID_STRIDE(i, n) {
    const float gi = g[i] + wd * p[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// loss += sum (pred - target)^2 / count; grad = 2 (pred - target) / count.
// One addition to the loss per block: with one per warp of a block per 256
// values, 32768 additions to one address took 53 us for 8 x 256 x 512 values
// and rounded the loss at each of them.
__global__ void __launch_bounds__(256) mse_kernel(long long n, const float* pred, const float* target, float inv_count,
                                                  float* grad, float* loss) {
  pdl_wait();
  pdl_trigger();
  __shared__ float part[8];
  float a = 0.f;
  GRID_STRIDE(i, n) {
    const float d = pred[i] - target[i];
    grad[i] = 2.f * d * inv_count;
    a += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) a += part[k];
    atomicAdd(loss, a * inv_count);
  }
}

}  // namespace

cudaError_t launch_to_chw(int n, int h, int w, int c, int cstride, int coff, const bf16* x, int copies, bf16* out,
                          cudaStream_t s) {
  const size_t smem = (size_t)(TCHW_X + 2) * c * sizeof(bf16);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(to_chw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)((w + TCHW_X - 1) / TCHW_X), (unsigned)(n * h));
  launch_nn(to_chw_kernel, grid, 256, smem, s, n, h, w, c, cstride, coff, x, copies, out);
  return cudaGetLastError();
}

cudaError_t launch_conv_in_fwd(int n, int h, int w, int c, const float* in, const float* W, const float* b, bf16* out,
                               int cstride, int coff, cudaStream_t s) {
  const long long threads = (long long)n * h * ((w + CIN_PX - 1) / CIN_PX);
  const int blocks = blocks_for(2 * threads);
  if (c <= 256)
    launch_nn(conv_in_fwd_kernel<true>, blocks, 128, (size_t)19 * c * 4, s, n, h, w, c, in, W, b, out, cstride, coff);
  else
    launch_nn(conv_in_fwd_kernel<false>, blocks, 128, 0, s, n, h, w, c, in, W, b, out, cstride, coff);
  return cudaGetLastError();
}

static long long vs_blocks(int n, int h, int w) {
  return (long long)n * ((h + VS_ROWS - 1) / VS_ROWS) * ((w + VS_X - 1) / VS_X);
}

cudaError_t launch_conv_in_wgrad(int n, int h, int w, int c, const float* in, const bf16* dy, int dy_cstride,
                                 float* dW, float* db, cudaStream_t s) {
  // 4 channel groups of 4 channels per block
  const dim3 grid((unsigned)vs_blocks(n, h, w), (unsigned)((c + 15) / 16));
  const bool vec = c % 4 == 0 && dy_cstride % 4 == 0 && (reinterpret_cast<uintptr_t>(dy) & 7u) == 0;
  auto kern = vec ? vec_scalar_wgrad_kernel<1, 2, true> : vec_scalar_wgrad_kernel<1, 2, false>;
  launch_nn(kern, grid, 256, 0, s, h, w, c, dy, dy_cstride, in, dW, db, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_conv_out_fwd(int n, int h, int w, int c, const bf16* in, int cstride, const float* W,
                                const float* b, float* out, cudaStream_t s) {
  if (c == 32 || c == 64) {
    const size_t smem = (size_t)(COUT_R + 2) * (COUT_TX + 2) * (c / 8) * 16 + (size_t)9 * c * 4;
    auto kern = c == 32 ? conv_out_tile_kernel<4> : conv_out_tile_kernel<8>;
    static bool set[2] = {false, false};
    if (!set[c == 64]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      set[c == 64] = true;
    }
    const long long blocks = (long long)n * ((h + COUT_R - 1) / COUT_R) * ((w + COUT_TX - 1) / COUT_TX);
    launch_nn(kern, (unsigned)blocks, COUT_TX, smem, s, n, h, w, in, cstride, W, b, out);
    return cudaGetLastError();
  }
  launch_nn(conv_out_fwd_kernel, blocks_for((long long)n * h * w), 256, 0, s, n, h, w, c, in, cstride, W, b, out);
  return cudaGetLastError();
}

cudaError_t launch_conv_out_bwd(int n, int h, int w, int c, const float* g, const float* W, const bf16* act,
                                int act_cstride, bf16* dx, float* dW, float* db, cudaStream_t s) {
  const size_t smem = (size_t)9 * c * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(conv_out_dgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  launch_nn(conv_out_dgrad_kernel, blocks_for((long long)n * h * ((w + COD_PX - 1) / COD_PX) * (c / 8)), 256, smem, s,
            n, h, w, c, g, W, act, act_cstride, dx);
  // 4 channel groups of 8 channels per block
  const dim3 grid((unsigned)vs_blocks(n, h, w), (unsigned)((c + 31) / 32));
  launch_nn(vec_scalar_wgrad_kernel<-1, 1, true>, grid, 256, 0, s, h, w, c, act, act_cstride, g, dW, nullptr, db);
  return cudaGetLastError();
}

cudaError_t launch_pool2(int n, int h, int w, int c, const bf16* in, int cs_in, int coff_in, bf16* out,
                         cudaStream_t s) {
  launch_nn(pool2_kernel, blocks_for((long long)n * (h / 2) * (w / 2) * (c / 8)), 256, 0, s,
            n, h, w, c, in, cs_in, coff_in, out);
  return cudaGetLastError();
}

cudaError_t launch_up2(int n, int h, int w, int c, const bf16* in, bf16* out, int cs_out, int coff_out,
                       cudaStream_t s) {
  launch_nn(up2_kernel, blocks_for((long long)n * h * w * (c / 8)), 256, 0, s, n, h, w, c, in, out, cs_out, coff_out);
  return cudaGetLastError();
}

cudaError_t launch_up2_bwd(int n, int h, int w, int c, const float* g, int cs_g, int coff_g, const bf16* act,
                           bf16* out, cudaStream_t s) {
  launch_nn(up2_bwd_kernel, blocks_for((long long)n * (h / 2) * (w / 2) * (c / 8)), 256, 0, s,
            n, h, w, c, g, cs_g, coff_g, act, out);
  return cudaGetLastError();
}

cudaError_t launch_pool2_bwd(int n, int h, int w, int c, const float* gp, const float* gs, int cs_s, int coff_s,
                             const bf16* act, int cs_a, int coff_a, bf16* out, cudaStream_t s) {
  launch_nn(pool2_bwd_kernel, blocks_for((long long)n * h * w * (c / 8)), 256, 0, s,
            n, h, w, c, gp, gs, cs_s, coff_s, act, cs_a, coff_a, out);
  return cudaGetLastError();
}

cudaError_t launch_bias_grad(int n, long long hw, int c, const bf16* dy, float* db, cudaStream_t s) {
  const dim3 grid(32, c);
  launch_nn(bias_grad_kernel, grid, 256, 0, s, n, hw, c, dy, db);
  return cudaGetLastError();
}

cudaError_t launch_bias_grad_nhwc(long long pixels, int c, const bf16* dy, float* db, cudaStream_t s) {
  if (c > 2048) return cudaErrorInvalidValue;  // one channel vector per thread
  long long b = (pixels * (c / 8) + 256 * 32 - 1) / (256 * 32);
  b = b > 152 * 8 ? 152 * 8 : b;
  launch_nn(bias_grad_nhwc_kernel, (unsigned)b, 256, (size_t)c * 4, s, pixels, c, dy, db);
  return cudaGetLastError();
}

cudaError_t launch_pack_weights(int cout, int cin, const float* W, bf16* wt, bf16* wflip, cudaStream_t s) {
  launch_nn(pack_weights_kernel, blocks_for((long long)cout * cin * 9), 256, 0, s, cout, cin, W, wt, wflip);
  return cudaGetLastError();
}

cudaError_t launch_adam(long long n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                        float eps, int step, float wd, cudaStream_t s) {
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  launch_nn(adam_kernel, blocks_for(n), 256, 0, s, n, p, g, m, v, lr, b1, b2, eps, c1, c2, wd);
  return cudaGetLastError();
}

cudaError_t launch_mse(long long n, const float* pred, const float* target, float* grad, float* loss,
                       cudaStream_t s) {
  const int b = blocks_for(n);
  launch_nn(mse_kernel, b < 152 * 4 ? b : 152 * 4, 256, 0, s, n, pred, target, 1.f / (float)n, grad, loss);
  return cudaGetLastError();
}

}  // namespace nn
}  // namespace sgb
