// Epilogue of the tensor-core convolutions: accumulator columns of one output
// pixel (TMEM lane) -> bias, ReLU, mask -> bf16 / fp32 NHWC stores.
#pragma once

#include <cuda_bf16.h>

#include "nn_args.cuh"
#include "tcgen05.cuh"

namespace sgb {
namespace nn {

// 16-byte store of eight bf16 values
__device__ __forceinline__ void st_bf16x8(__nv_bfloat16* p, const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
// 32-byte (whole-sector) store of eight fp32 values
__device__ __forceinline__ void st_f32x8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// Columns [taddr, taddr + BN) of this thread's lane are output channels n0 ..
// of pixel `pix`; every lane of the warp calls it (tcgen05.ld is a warp
// collective), only those with `inrow` store.
template <int BN>
__device__ __forceinline__ void conv_epilogue(const GemmArgs& g, uint32_t taddr, int n0, long long pix, bool inrow) {
  const bool vb = ((g.out_cstride | g.out_coff) & 7) == 0;
  const bool vf = ((g.out_cstride | g.out_coff) & 3) == 0;
  const bool vf8 = vb && (reinterpret_cast<uintptr_t>(g.out_f32) & 31u) == 0;
  const bool vm = (g.mask_cstride & 7) == 0;
#pragma unroll 1
  for (int c = 0; c < BN; c += 16) {
    float v[16];
    tmem_ld16(taddr + c, v);
    const int co = n0 + c;
    if (!inrow || co >= g.Cout) continue;
    const bool whole = co + 16 <= g.Cout;
    if (g.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += (co + j < g.Cout) ? g.bias[co + j] : 0.f;
    }
    if (g.relu) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = v[j] < 0.f ? 0.f : v[j];
    }
    if (g.mask != nullptr) {
      const __nv_bfloat16* mp = g.mask + pix * g.mask_cstride + co;
      if (whole && vm) {
        const uint4 m0 = *reinterpret_cast<const uint4*>(mp);
        const uint4 m1 = *reinterpret_cast<const uint4*>(mp + 8);
        const __nv_bfloat16* mb0 = reinterpret_cast<const __nv_bfloat16*>(&m0);
        const __nv_bfloat16* mb1 = reinterpret_cast<const __nv_bfloat16*>(&m1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = __bfloat162float(mb0[j]) > 0.f ? v[j] : 0.f;
          v[8 + j] = __bfloat162float(mb1[j]) > 0.f ? v[8 + j] : 0.f;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (co + j < g.Cout) v[j] = __bfloat162float(mp[j]) > 0.f ? v[j] : 0.f;
      }
    }
    if (g.out_f32 != nullptr) {
      float* o = g.out_f32 + pix * g.out_cstride + g.out_coff + co;
      if (whole && vf8) {
        st_f32x8(o, v);
        st_f32x8(o + 8, v + 8);
      } else if (whole && vf) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (co + j < g.Cout) o[j] = v[j];
      }
    }
    if (g.out_bf16 != nullptr) {
      __nv_bfloat16* o = g.out_bf16 + pix * g.out_cstride + g.out_coff + co;
      if (whole && vb) {
        st_bf16x8(o, v);
        st_bf16x8(o + 8, v + 8);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (co + j < g.Cout) o[j] = __float2bfloat16_rn(v[j]);
      }
    }
  }
}

}  // namespace nn
}  // namespace sgb
