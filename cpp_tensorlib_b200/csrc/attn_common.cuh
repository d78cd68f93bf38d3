// Lane-to-dims mapping and key-row loads shared by the decode and the prefill attention
// kernels, for f32 and bf16 caches; one row of bf16 attention in plain f32.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace tlb {

// first dim of a lane's j-th float4 of q / acc / a key row
template <int LPK, bool BF>
__device__ __forceinline__ int attn_dim0(int sub, int j) {
  return BF ? 8 * (sub + LPK * (j >> 1)) + 4 * (j & 1) : 4 * (sub + LPK * j);
}
// the lane's CH float4 of one key row held in a tile (f32 as it is, bf16 widened)
template <int D, int LPK, int CH, bool BF>
__device__ __forceinline__ void attn_load_row(const unsigned char* row, int sub, float4 (&kv)[CH]) {
  if (BF) {
#pragma unroll
    for (int jj = 0; jj < CH / 2; jj++) {
      const uint4 w = *(const uint4*)(row + (size_t)(sub + LPK * jj) * 16);
      kv[2 * jj] = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u),
                               __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
      kv[2 * jj + 1] = make_float4(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u),
                                   __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
    }
  } else {
#pragma unroll
    for (int j = 0; j < CH; j++) kv[j] = *(const float4*)(row + (size_t)(sub + LPK * j) * 16);
  }
}

// A query over rows k0, k0 + step, .. below k1 of a bf16 head by one warp, a key at a time in plain f32 (D / 32
// dimensions a lane): for results that came out NaN on the tensor pipe.  There a query or a weight enters as three planes,
// and an infinite key or value gives infinity less infinity, or infinity times a plane's zero, where f32 has one infinite
// product; and a key that only later rows of a tile see counts as zero times its value.  A key whose score is -infinity
// has no weight.  `scale` with log2(e).  Not inlined: it runs next to never, and the kernels keep their registers.
template <int D>
struct AttnRow {
  float acc[D / 32], m, l;
};
template <int D>
__device__ __noinline__ AttnRow<D> attn_row_again(const float* q, const __nv_bfloat16* K, const __nv_bfloat16* V,
                                                  float scale, int k0, int k1, int step) {
  constexpr int N = D / 32;
  const int lane = threadIdx.x & 31;
  AttnRow<D> a;
  float x[N];
#pragma unroll
  for (int i = 0; i < N; i++) {
    x[i] = q[lane * N + i] * scale;
    a.acc[i] = 0.f;
  }
  a.m = -INFINITY;
  a.l = 0.f;
  for (int j = k0; j < k1; j += step) {
    const __nv_bfloat16 *k = K + (size_t)j * D + lane * N, *v = V + (size_t)j * D + lane * N;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; i++) s = fmaf(x[i], __bfloat162float(k[i]), s);
    s = warp_sum(s);
    if (s == -INFINITY) continue;
    if (s > a.m) {
      const float f = exp2f(a.m - s);
      a.l *= f;
#pragma unroll
      for (int i = 0; i < N; i++) a.acc[i] *= f;
      a.m = s;
    }
    const float p = exp2f(s - a.m);
    a.l += p;
#pragma unroll
    for (int i = 0; i < N; i++) a.acc[i] = fmaf(p, __bfloat162float(v[i]), a.acc[i]);
  }
  return a;
}

}  // namespace tlb
