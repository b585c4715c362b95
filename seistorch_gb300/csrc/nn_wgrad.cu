// Weight gradient of a 3x3 convolution on the 5th-generation tensor cores,
// straight from the NHWC activations:
//   dW[co][ci][ky][kx] += sum_p x[p + (ky - 1, kx - 1)][ci] dy[p][co].
//
// K is the pixels.  In NHWC a pixel's channels are contiguous, so both
// operands are "MN-major": a panel of 64 channels (128-byte rows, 128-byte
// swizzle; 32 channels in 64-byte rows where cout is 32) by 64 pixels is one
// TMA box, and no channel-major copies are needed.  A CTA takes one tap row
// ky, 128 input channels (A, two panels), BN output channels (B) and a range
// of 64-pixel chunks.  The A box carries one pixel of halo on each side; the
// three taps kx of the row read the same box from a start address one pixel
// row (128 bytes) further each, the swizzle pattern still starting at the
// panel's 1024-byte boundary, into three accumulators of BN columns.  Border
// taps read TMA's zero fill.
//
// The pixels are split as in the channel-major kernel (sgb_nn_conv3x3_wgrad):
// the tensor cores' accumulation over a split is the coarsest rounding of the
// path, so a split's sum here is that kernel's, and only the order of the
// splits' fp32 additions is open, there as here.  Layers of few splits take one
// tap and 32 or 64 output channels per CTA instead, to fill the SMs.
//
// What bounds it: the read of A from shared memory (128 x 16 per MMA whatever
// BN is) and the L2 reads of x (three tap rows); the channel-major form also
// writes and reads a transposed dy and three column-shifted transposes of x,
// and reads x nine times.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "sgb_common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"
#include "nn_args.cuh"

namespace sgb {
namespace nn {
namespace {

constexpr int WG_PX = 64;                  // pixels per K step
constexpr int WG_A_ROWS = WG_PX + 2;       // with the halo of the kx taps
constexpr int WG_A_PANEL = 9216;           // 66 rows of 128 bytes, to the next 1024
template <int BN, int TAPS, bool ALONE>
struct WgLayout {
  static constexpr int RB = BN >= 64 ? 128 : 64;  // bytes of a B row
  static constexpr int B_PANELS = BN >= 64 ? BN / 64 : 1;
  static constexpr int B_PANEL = WG_PX * RB;
  static constexpr int STAGE = 2 * WG_A_PANEL + B_PANELS * B_PANEL;
  // stages: about 200 KB where a CTA has the SM alone (eight steps in flight:
  // a step's copies take about two steps' time to arrive), half where two share it
  static constexpr int S = BN == 128 ? 6 : (ALONE ? 8 : 4);
  static constexpr int BYTES = S * STAGE + 1024 + 256;
  static constexpr int COLS = TAPS == 1 ? BN : (BN == 128 ? 512 : (BN == 64 ? 256 : 128));  // TAPS BN, to a power of two
};

// MN-major operand descriptor: panels `lbo` bytes apart, 8-pixel groups `sbo` bytes apart.
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint64_t layout) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) |
         (layout << 61);
}

template <int BN, int TAPS, bool ALONE>
__global__ void __launch_bounds__(128) nn_wgrad_kernel(const __grid_constant__ CUtensorMap tmX,
                                                       const __grid_constant__ CUtensorMap tmD, const WgradArgs g) {
  using Lay = WgLayout<BN, TAPS, ALONE>;
  constexpr int S = Lay::S;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + S * Lay::STAGE);
  uint64_t* empty = full + S;
  uint64_t* acc = empty + S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc + 1);
  __shared__ int s_fail, s_issued, s_consumed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) tmem_alloc(tmem_slot, Lay::COLS);
  if (threadIdx.x == 32) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc, 1);
    fence_mbar_init();
    s_fail = s_issued = s_consumed = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // the barriers and the TMEM are set up beside the previous launch
  pdl_wait();
  pdl_trigger();
  volatile int* fail = &s_fail;
  constexpr int GROUPS = 9 / TAPS;  // tap rows, or single taps
  const int tap0 = (blockIdx.y % GROUPS) * TAPS, ky = tap0 / 3, kx0 = tap0 - 3 * ky;
  const int m0 = (blockIdx.y / GROUPS) * 128, n0 = blockIdx.z * BN;
  const int k0 = blockIdx.x * g.k_per_split, k1 = min(k0 + g.k_per_split, g.kiters);
  const int panels = g.Cin - m0 > 64 ? 2 : 1;  // rows beyond Cin: not loaded, their sums not stored

  if (warp == 0) {
    const uint32_t el = elect_one();
    int xc = k0 % g.wchunks, y = k0 / g.wchunks % g.H, n = k0 / g.wchunks / g.H, it = 0;
    for (int k = k0; k < k1; ++k, ++it) {
      const int s = it % S;
      // warp-uniform, one lane issues
      if (!__all_sync(0xffffffffu, !*fail && (it < S || mbar_wait(&empty[s], ((it / S) - 1) & 1, g.status)))) {
        *fail = 1;
        break;
      }
      if (el) {
        unsigned char* sa = base + s * Lay::STAGE;
        unsigned char* sb = sa + 2 * WG_A_PANEL;
        mbar_arrive_expect_tx(&full[s], panels * WG_A_ROWS * 128 + Lay::B_PANELS * Lay::B_PANEL);
        tma_load_4d(sa, &tmX, m0, xc * WG_PX - 1, y + ky - 1, n, &full[s]);
        if (panels > 1) tma_load_4d(sa + WG_A_PANEL, &tmX, m0 + 64, xc * WG_PX - 1, y + ky - 1, n, &full[s]);
#pragma unroll
        for (int p = 0; p < Lay::B_PANELS; ++p)
          tma_load_4d(sb + p * Lay::B_PANEL, &tmD, n0 + 64 * p, xc * WG_PX, y, n, &full[s]);
      }
      if (++xc == g.wchunks) {
        xc = 0;
        if (++y == g.H) {
          y = 0;
          ++n;
        }
      }
    }
    if (lane == 0) s_issued = it;
  } else if (warp == 1) {
    const uint32_t el = elect_one();
    const uint32_t idesc = mma_idesc_bf16(128, BN) | (1u << 15) | (1u << 16);  // A and B MN-major
    int it = 0;
    for (int k = k0; k < k1; ++k, ++it) {
      const int s = it % S;
      // warp-uniform: the MMAs are issued by one lane of a converged warp
      if (!__all_sync(0xffffffffu, !*fail && mbar_wait(&full[s], (it / S) & 1, g.status))) {
        *fail = 1;
        break;
      }
      tc_fence_after();
      const uint32_t sa = smem_u32(base + s * Lay::STAGE), sb = sa + 2 * WG_A_PANEL;
      const uint64_t da = mn_desc(sa, WG_A_PANEL, 1024, 2);
      const uint64_t db = Lay::RB == 128 ? mn_desc(sb, Lay::B_PANEL, 1024, 2) : mn_desc(sb, Lay::B_PANEL, 512, 4);
#pragma unroll
      for (int t = 0; t < TAPS; ++t)
#pragma unroll
        for (int kk = 0; kk < WG_PX / 16; ++kk)
          mma_bf16(el, tmem + t * BN, da + (uint64_t)(((kx0 + t) * 128 + kk * 2048) >> 4),
                   db + (uint64_t)((kk * 16 * Lay::RB) >> 4), idesc, (k > k0 || kk > 0) ? 1u : 0u);
      mma_commit(el, &empty[s]);
    }
    if (lane == 0) s_consumed = it;
    mma_commit(el, acc);  // completes once every MMA issued above has finished
  }
  __syncthreads();
  const bool done = __all_sync(0xffffffffu, mbar_wait(acc, 0, g.status));
  if (threadIdx.x == 0 && *fail)
    for (int i = s_consumed; i < s_issued; ++i) mbar_wait(&full[i % S], (i / S) & 1, nullptr);
  tc_fence_after();
  if (done && !*fail && k1 > k0) {
    const int ci = m0 + warp * 32 + lane;  // TMEM lane == accumulator row
    const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int c = 0; c < BN; c += 16) {
      float v[TAPS][16];
#pragma unroll
      for (int t = 0; t < TAPS; ++t) tmem_ld16(taddr + t * BN + c, v[t]);
      if (ci >= g.Cin) continue;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int co = n0 + c + j;
        if (co >= g.Cout) break;
        float* o = g.dw + ((long long)co * g.Cin + ci) * 9 + tap0;
#pragma unroll
        for (int t = 0; t < TAPS; ++t) atomicAdd(o + t, v[t][j]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, Lay::COLS);
  }
}

int sm_count() {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int BN, int TAPS, bool ALONE>
cudaError_t launch_s(const CUtensorMap* maps, const WgradArgs& g, int splits, cudaStream_t s) {
  using Lay = WgLayout<BN, TAPS, ALONE>;
  auto kern = nn_wgrad_kernel<BN, TAPS, ALONE>;
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::BYTES);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    set = true;
  }
  const dim3 grid((unsigned)splits, (unsigned)(9 / TAPS * ((g.Cin + 127) / 128)), (unsigned)((g.Cout + BN - 1) / BN));
  return launch_pdl(kern, dim3(grid), dim3(128), Lay::BYTES, s, maps[0], maps[1], g);
}

template <int BN, int TAPS>
cudaError_t launch_t(const CUtensorMap* maps, const WgradArgs& g, int splits, cudaStream_t s) {
  const long long ctas = (long long)splits * (9 / TAPS) * ((g.Cin + 127) / 128) * ((g.Cout + BN - 1) / BN);
  return ctas <= sm_count() ? launch_s<BN, TAPS, true>(maps, g, splits, s) : launch_s<BN, TAPS, false>(maps, g, splits, s);
}

}  // namespace

// Output channels per tile and taps per CTA of least estimated time.  Cycles of
// a step measured at the layers' sizes (batch 8 of 256 x 512): 62 / 78 per MMA
// of 32 / 64 output channels, and about 600 where the copies' latency, not the
// MMAs, is what a step waits for (one tap).  128 -> 128 channels: 64 us as three
// taps by 64, 40 us as one tap by 64; 384 -> 128: 162 us as one tap by 128 in
// two waves, 75 us as three taps by 64 in one.  Against the best variant of each of
// the nine layers the rule is 9 % off at batch 8 of 256 x 512 (729 us in all), 9 and
// 12 % at batch 1 and 2, 0.5 % at 4 of 384 x 1024 and 8 % at 8 of 128 x 512.  The B
// box of the tensor map is 64 channels (32 for bn = 32).
static void wgrad_tile(const WgradArgs& g, int splits, int* bn, int* taps) {
  const int sms = sm_count(), mt = (g.Cin + 127) / 128;
  int best = 0;
  for (int t : {3, 1})
    for (int n : {128, 64, 32}) {
      if (n > 32 && g.Cout <= n / 2) continue;  // half the tile empty
      const int ctas = splits * (9 / t) * mt * ((g.Cout + n - 1) / n), mma = 4 * t * (46 + n / 2);
      const int cost = (ctas + sms - 1) / sms * (mma > 600 ? mma : 600);
      if (best == 0 || cost < best) {
        best = cost;
        *bn = n;
        *taps = t;
      }
    }
}

static int wgrad_splits(const WgradArgs& g, int* per) {
  int splits = (g.kiters + 127) / 128;
  if (splits > 64) splits = 64;
  *per = (g.kiters + splits - 1) / splits;
  return (g.kiters + *per - 1) / *per;
}

int wgrad_bn(const WgradArgs& g) {
  int per, bn, taps;
  const int splits = wgrad_splits(g, &per);
  wgrad_tile(g, splits, &bn, &taps);
  return bn;
}

cudaError_t launch_wgrad(const CUtensorMap* maps, const WgradArgs& g0, cudaStream_t s) {
  WgradArgs g = g0;
  int bn, taps;
  const int splits = wgrad_splits(g, &g.k_per_split);
  wgrad_tile(g, splits, &bn, &taps);
  if (taps == 3) {
    switch (bn) {
      case 32: return launch_t<32, 3>(maps, g, splits, s);
      case 64: return launch_t<64, 3>(maps, g, splits, s);
      case 128: return launch_t<128, 3>(maps, g, splits, s);
    }
  } else {
    switch (bn) {
      case 32: return launch_t<32, 1>(maps, g, splits, s);
      case 64: return launch_t<64, 1>(maps, g, splits, s);
      case 128: return launch_t<128, 1>(maps, g, splits, s);
    }
  }
  return cudaErrorInvalidValue;
}

}  // namespace nn
}  // namespace sgb
