// 3x3 convolution of an NHWC image on the tensor cores for layers whose weights
// fit in shared memory (the preconditioner's two finer levels, forward and data
// gradient): implicit GEMM with the input rows kept on chip.
//
// A persistent CTA holds the weights of all nine taps, loaded once, and walks
// down a strip of 128 columns.  Each step loads one new input row (130 pixels:
// the strip and one of halo on either side, all channels; TMA zero fill is the
// padding) into a ring of R row slots and computes one 128-pixel row of outputs
// from the last three.  The three taps kx of a row read the same slot from a
// start address one pixel further each: the rows of a K-major operand are RB
// bytes, the swizzle pattern starts at the panel's 1024-byte boundary and is a
// function of the address.  Accumulation order as in nn_gemm_kernel (tap,
// channel chunk, 16 channels), so the sums are the same.
//
//   warp 0 -- TMA producer; warp 1 -- MMA issuer into accumulator
//   (tile & 1); warps 2..5 -- epilogue of the finished accumulator.
// Every wait is bounded; on a timeout the CTA records it, drains what it issued
// and frees its TMEM.
//
// What bounds it: the read of A from shared memory (128 x 16 per MMA) for 96
// input channels, the stores for 96 fp32 outputs, DRAM for 32 channels.  With
// one input box per tap (nn_gemm_kernel) the input is read nine times through
// L2 and the weights once per 128 outputs.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "sgb_common.cuh"
#include "tma.cuh"
#include "nn_epilogue.cuh"
#include "row_ring.cuh"

namespace sgb {
namespace nn {
namespace {

constexpr int CR_MAX_SLOTS = 8;
constexpr int CR_SMEM = 224 * 1024;
// A CTA's range of output rows pays two extra input rows and the weights: at
// least four rows each.
constexpr int CR_MIN_TILES = 4;

template <int BN, int RB>
struct RowLayout {
  static constexpr int PANEL = RB == 128 ? 17408 : 9216;  // 130 pixel rows, to the next 1024
  static constexpr int W_PANEL = BN * RB;                 // one tap, one channel chunk
  static constexpr int ACC = BN < 32 ? 32 : BN;
  static constexpr int COLS = 2 * ACC <= 64 ? 64 : (2 * ACC <= 128 ? 128 : 256);
};

template <int BN, int RB>
__global__ void __launch_bounds__(192) nn_conv_row_kernel(const __grid_constant__ CUtensorMap tmX,
                                                          const __grid_constant__ CUtensorMap tmW, const GemmArgs g,
                                                          const int R) {
  using Lay = RowLayout<BN, RB>;
  constexpr int KSTEPS = RB / 32;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int slot_bytes = g.nchunk * Lay::PANEL, w_bytes = 9 * g.nchunk * Lay::W_PANEL;
  unsigned char* rows = base + w_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(rows + R * slot_bytes);
  uint64_t* empty = full + CR_MAX_SLOTS;
  uint64_t* acc_full = empty + CR_MAX_SLOTS;  // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint64_t* wfull = acc_empty + 2;
  uint64_t* done = wfull + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  __shared__ int s_fail, s_issued, s_consumed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) tmem_alloc(tmem_slot, Lay::COLS);
  if (threadIdx.x == 32) {
    for (int s = 0; s < R; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);  // one arrival per epilogue warp
    }
    mbar_init(wfull, 1);
    mbar_init(done, 1);
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
  // tiles in the order image, strip, row (rows fastest); this CTA's range
  const long long ntiles = (long long)g.N * g.tiles_x * g.H;
  const int t0 = (int)(ntiles * blockIdx.x / gridDim.x), t1 = (int)(ntiles * (blockIdx.x + 1) / gridDim.x);

  if (warp == 0) {  // all lanes run the loop, one issues
    const uint32_t el = elect_one();
    if (el) {
      mbar_arrive_expect_tx(wfull, w_bytes);
      for (int tap = 0; tap < 9; ++tap)
        for (int c = 0; c < g.nchunk; ++c)
          tma_load_3d(base + (tap * g.nchunk + c) * Lay::W_PANEL, &tmW, c * (RB / 2), tap, 0, wfull);
    }
    int r = 0;  // rows loaded
    bool ok = true;
    for (int t = t0; t < t1 && ok; ++t) {
      const int y = t % g.H, st = t / g.H;
      const int x = (st % g.tiles_x) * 128 - 1, n = st / g.tiles_x;
      for (int yy = (t == t0 || y == 0) ? y - 1 : y + 1; yy <= y + 1; ++yy, ++r) {
        const int s = r % R;
        ok = __all_sync(0xffffffffu, !*fail && (r < R || mbar_wait(&empty[s], ((r / R) - 1) & 1, g.status)));
        if (!ok) break;
        if (el) {
          mbar_arrive_expect_tx(&full[s], g.nchunk * 130 * RB);
          for (int c = 0; c < g.nchunk; ++c)
            tma_load_4d(rows + s * slot_bytes + c * Lay::PANEL, &tmX, c * (RB / 2), x, yy, n, &full[s]);
        }
      }
    }
    if (!ok) *fail = 1;
    if (lane == 0) s_issued = r;
  } else if (warp == 1) {
    const uint32_t el = elect_one();
    const uint32_t idesc = mma_idesc_bf16(128, BN);
    const uint32_t wbase = smem_u32(base), rbase = smem_u32(rows);
    int r = 0;  // rows that have arrived
    // every decision is warp-uniform: the MMAs are issued by one lane of a converged warp
    auto wait = [&](uint64_t* bar, int parity) -> bool {
      return __all_sync(0xffffffffu, !*fail && mbar_wait(bar, parity, g.status));
    };
    bool ok = wait(wfull, 0);
    for (int t = t0, lt = 0; t < t1 && ok; ++t, ++lt) {
      const int y = t % g.H, buf = lt & 1;
      const int need = (t == t0 || y == 0) ? 3 : 1;
      ok = take_rows(need, r, [&](int row) { return wait(&full[row % R], (row / R) & 1); });
      if (ok && lt >= 2) ok = wait(&acc_empty[buf], ((lt >> 1) - 1) & 1);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)(buf * Lay::ACC);
      for (int ky = 0; ky < 3; ++ky) {
        const uint64_t da0 = smem_desc<RB>(rbase + (uint32_t)(((r - 3 + ky) % R) * slot_bytes));
        const uint64_t db0 = smem_desc<RB>(wbase + (uint32_t)(ky * 3 * g.nchunk * Lay::W_PANEL));
#pragma unroll
        for (int kx = 0; kx < 3; ++kx)
          for (int c = 0; c < g.nchunk; ++c) {
            const uint64_t da = da0 + (uint64_t)((c * Lay::PANEL + kx * RB) >> 4);
            const uint64_t db = db0 + (uint64_t)(((kx * g.nchunk + c) * Lay::W_PANEL) >> 4);
#pragma unroll
            for (int kk = 0; kk < KSTEPS; ++kk)
              mma_bf16(el, d, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), idesc,
                       (kx > 0 || kk > 0) ? 1u : (uint32_t)(ky + c));
          }
      }
      // the row above is done with; the strip's last tile is done with all three
      mma_commit(el, &empty[(r - 3) % R]);
      if (y == g.H - 1) {
        mma_commit(el, &empty[(r - 2) % R]);
        mma_commit(el, &empty[(r - 1) % R]);
      }
      mma_commit(el, &acc_full[buf]);
    }
    if (!ok) *fail = 1;
    if (lane == 0) s_consumed = r;
    mma_commit(el, done);  // completes once every MMA issued above has finished
  } else if (warp >= 2) {
    const int quarter = warp & 3;  // TMEM lanes 32 (warp % 4) .. + 31
    for (int t = t0, lt = 0; t < t1; ++t, ++lt) {
      const int y = t % g.H, st = t / g.H, buf = lt & 1;
      const int x = (st % g.tiles_x) * 128 + quarter * 32 + lane;
      // the decision is warp-uniform (tcgen05.ld is a warp collective)
      const bool got = __all_sync(0xffffffffu, !*fail && mbar_wait(&acc_full[buf], (lt >> 1) & 1, g.status));
      if (!got) {
        *fail = 1;
        break;
      }
      tc_fence_after();
      const long long pix = ((long long)(st / g.tiles_x) * g.H + y) * g.W + x;
      conv_epilogue<BN>(g, tmem + (uint32_t)(buf * Lay::ACC) + ((uint32_t)(quarter * 32) << 16), 0, pix, true);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 32) mbar_wait(done, 0, nullptr);
  if (threadIdx.x == 0 && *fail) {  // boxes issued but never consumed
    mbar_wait(wfull, 0, nullptr);
    for (int i = s_consumed; i < s_issued; ++i) mbar_wait(&full[i % R], (i / R) & 1, nullptr);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, Lay::COLS);
  }
}

// CTAs per SM and row slots for nchunk channel chunks: as many CTAs as fit
// with four slots each (three rows in use, one in flight) and at most four,
// then the slots that the shared memory leaves.  0 if one CTA does not fit.
template <int BN, int RB>
int plan_row(int nchunk, int* slots, int* smem) {
  using Lay = RowLayout<BN, RB>;
  const int fixed = 9 * nchunk * Lay::W_PANEL + 1024 + 256, slot = nchunk * Lay::PANEL;
  int per = 512 / Lay::COLS;
  if (per > 4) per = 4;
  for (; per >= 1; --per) {
    const int room = CR_SMEM / per - 1024 - fixed;
    if (room < 4 * slot) continue;
    *slots = room / slot < CR_MAX_SLOTS ? room / slot : CR_MAX_SLOTS;
    *smem = fixed + *slots * slot;
    // no more CTAs than their accumulators allow: TMEM allocation would wait
    if ((512 / Lay::COLS + 1) * (*smem + 1024) <= CR_SMEM) *smem = CR_SMEM / (512 / Lay::COLS + 1) + 1;
    return per;
  }
  return 0;
}

template <int BN, int RB>
cudaError_t launch_row_t(const CUtensorMap* maps, const GemmArgs& g, cudaStream_t s) {
  auto kern = nn_conv_row_kernel<BN, RB>;
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CR_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    set = true;
  }
  int dev = 0, sms = 152, R = 0, smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int per = plan_row<BN, RB>(g.nchunk, &R, &smem);
  if (per == 0) return cudaErrorInvalidValue;
  const long long ntiles = (long long)g.N * g.tiles_x * g.H;
  const long long cap = (long long)per * sms, most = ntiles / CR_MIN_TILES;
  return launch_pdl(kern, dim3((unsigned)(most < cap ? most : cap)), dim3(192), smem, s, maps[0], maps[1], g, R);
}

template <int RB>
int plan_rb(int bn, int nchunk) {
  int a, b;
  switch (bn) {
    case 32: return plan_row<32, RB>(nchunk, &a, &b);
    case 64: return plan_row<64, RB>(nchunk, &a, &b);
    case 96: return plan_row<96, RB>(nchunk, &a, &b);
    case 128: return plan_row<128, RB>(nchunk, &a, &b);
  }
  return 0;
}

template <int RB>
cudaError_t launch_rb(int bn, const CUtensorMap* maps, const GemmArgs& g, cudaStream_t s) {
  switch (bn) {
    case 32: return launch_row_t<32, RB>(maps, g, s);
    case 64: return launch_row_t<64, RB>(maps, g, s);
    case 96: return launch_row_t<96, RB>(maps, g, s);
    case 128: return launch_row_t<128, RB>(maps, g, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

// Output channels per tile (all of them) if the layer can keep its weights and
// rows on chip, else 0.  Below CR_MIN_TILES rows of 128 pixels for each SM the
// CTAs of nn_gemm_kernel, one tile each, fill the GPU better.
int conv_row_bn(const GemmArgs& g, int rb) {
  if (g.W % 128 != 0 || g.Cout > 128) return 0;
  const int bn = (g.Cout + 31) / 32 * 32;
  const int per = rb == 128 ? plan_rb<128>(bn, g.nchunk) : plan_rb<64>(bn, g.nchunk);
  if (per == 0) return 0;
  const long long ntiles = (long long)g.N * (g.W / 128) * g.H;
  if (ntiles >= (1LL << 30) || ntiles < 152LL * CR_MIN_TILES) return 0;
  return bn;
}

cudaError_t launch_conv_row(int bn, int rb, const CUtensorMap* maps, const GemmArgs& g, cudaStream_t s) {
  return rb == 128 ? launch_rb<128>(bn, maps, g, s) : launch_rb<64>(bn, maps, g, s);
}

}  // namespace nn
}  // namespace sgb
