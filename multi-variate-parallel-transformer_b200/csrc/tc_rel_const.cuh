// Pre-kernel shared by the tensor-core forward and backward: the bias halves of the two relative
// products, which do not depend on the query.
#pragma once

#include <cuda_bf16.h>

#include "tc_ptx.cuh"

namespace mvpa {

// Per-column constants of the two relative products, once per kv head instead of once per CTA:
//   relc[hk][j] = vt[hk] . r_time[hk][j]  (j < T),   relc[hk][128 + j] = z[hk] . r_chan[hk][j]  (j < C)
// (the bias halves of `_rel_bias`, `attentions/attn.py:1308-1313`).
// One thread per column: its key row comes in with 16-byte loads that are all in flight at once (D is 64
// or 128 on the tensor-core paths: 8 or 16 loads), so the kernel costs one memory round trip, not D / 2.
// (`FLIGHT` of the row's 16-byte loads in flight at once; a kernel that is much else beside takes a few, for its size)
template <int D, int FLIGHT = D / 8>
static __device__ __forceinline__ float rel_const(const __nv_bfloat16* __restrict__ vt, const __nv_bfloat16* __restrict__ z,
                                                   const __nv_bfloat16* __restrict__ rt, const __nv_bfloat16* __restrict__ rc,
                                                   int T, int C, int hk, int column) {
  const int j = column & 127;
  const bool is_t = column < 128;
  const int rows = is_t ? T : C;
  float acc = 0.f;
  if (j < rows) {
    const uint4* key = reinterpret_cast<const uint4*>((is_t ? rt : rc) + ((size_t)hk * rows + j) * D);
    const uint4* bias = reinterpret_cast<const uint4*>((is_t ? vt : z) + (size_t)hk * D);
#pragma unroll 1
    for (int i0 = 0; i0 < D / 8; i0 += FLIGHT) {
      uint4 k[FLIGHT], b[FLIGHT];
#pragma unroll
      for (int i = 0; i < FLIGHT; ++i) {
        k[i] = key[i0 + i];
        b[i] = bias[i0 + i];
      }
#pragma unroll
      for (int i = 0; i < FLIGHT; ++i) {
        const uint32_t kw[4] = {k[i].x, k[i].y, k[i].z, k[i].w}, bw[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // the same pairs in the same order as a two-element walk over d
          const float ax = __uint_as_float(kw[e] << 16), ay = __uint_as_float(kw[e] & 0xffff0000u);
          const float bx = __uint_as_float(bw[e] << 16), by = __uint_as_float(bw[e] & 0xffff0000u);
          acc += ax * bx + ay * by;
        }
      }
    }
  }
  return acc;
}
template <int D>
static __device__ __forceinline__ void rel_const_row(const __nv_bfloat16* __restrict__ vt, const __nv_bfloat16* __restrict__ z,
                                                      const __nv_bfloat16* __restrict__ rt, const __nv_bfloat16* __restrict__ rc,
                                                      float* __restrict__ relc, int T, int C, int hk) {  // 256 threads
  relc[hk * 256 + threadIdx.x] = rel_const<D>(vt, z, rt, rc, T, C, hk, threadIdx.x);
}

template <int D>
static __global__ void __launch_bounds__(256) rel_const_kernel(const __nv_bfloat16* __restrict__ vt,
                                                               const __nv_bfloat16* __restrict__ z,
                                                               const __nv_bfloat16* __restrict__ rt,
                                                               const __nv_bfloat16* __restrict__ rc,
                                                               float* __restrict__ relc, int T, int C,
                                                               int* __restrict__ status_words) {
  ptx::griddep_launch();  // the next kernel's CTAs may come up; they wait for this grid's end before reading anything
  // (also clears the 64 status words of the kernels that follow: one memset node less in front of them)
  if (blockIdx.x == 0 && threadIdx.x < 64) status_words[threadIdx.x] = 0;
  rel_const_row<D>(vt, z, rt, rc, relc, T, C, blockIdx.x);
}

}  // namespace mvpa
