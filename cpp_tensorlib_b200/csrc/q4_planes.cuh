// Activation rows as the int4 tensor-core product reads them (gemm_q4_tc2.cu): two fp16 planes, hi and lo of
// x * 2^-e with one power of two e a row, and the row's 2^e.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace tlb {

struct Q4Planes {
  __half *hi, *lo;    // [M][K], K % 8 == 0
  float* rowscale;    // [M]
};
// planes of M rows of K inside `scratch` (gemm_q4_tc2_scratch_bytes(M, K) bytes, 16-byte aligned)
inline Q4Planes q4_planes_at(void* scratch, int M, int K) {
  Q4Planes p;
  p.hi = (__half*)scratch;
  p.lo = p.hi + (size_t)M * K;
  p.rowscale = (float*)(((uintptr_t)(p.lo + (size_t)M * K) + 255) & ~(uintptr_t)255);
  return p;
}

size_t gemm_q4_tc2_scratch_bytes(int M, int K);
constexpr size_t Q4_FEW_BYTES = (size_t)4 << 20;   // a context's planes for products of up to 8 rows
// The product's own scratch (`work`): the context's or a decoder's, for one product at a time.  Its first bytes
// (Q4_TICKET_BYTES) are zero before a product, and the product leaves them zero.
constexpr int Q4_TICKET_BYTES = 4096;   // room for 1024 SMs
size_t gemm_q4_work_bytes(int sm_count);
// whether a product of M rows takes the planes (and not another kernel), whether it could
bool gemm_q4_planes_eligible(const void* qw, const void* scales, int N, int K, int M);
bool gemm_q4_planes_possible(const void* qw, const void* scales, int N, int K, int M);
int gemm_q4_planes_launch(DeviceCtx* c, const Q4Planes& x, int M, const void* qw, const float* scales, float* y,
                          long long ldy, int N, int K, float alpha, float beta, void* work, cudaStream_t stream);
// x f32 rows -> planes, on a device of `sms` SMs
int launch_split_rows(const float* x, long long ldx, int M, int K, const Q4Planes& pl, int sms, cudaStream_t stream);

#ifdef __CUDACC__

// e of a row whose largest magnitude is mx: the scaled row stays below 2^14
__device__ __forceinline__ int q4_row_exponent(float mx) {
  if (!(mx > 0.f && mx < 3.0e38f)) return 0;
  int ex;
  frexpf(mx, &ex);            // mx = f * 2^ex, f in [0.5, 1)
  const int e = ex - 14;
  return e < -100 ? -100 : (e > 100 ? 100 : e);
}
// Eight consecutive k, scaled by s, as 16 bytes of each plane, in the order 0,4,1,5,2,6,3,7 -- the order in
// which the product's converters' nibble extraction lays out the weights.
__device__ __forceinline__ void q4_split8(const float4 a, const float4 b, float s, uint4& hi, uint4& lo) {
  const float f[8] = {a.x * s, b.x * s, a.y * s, b.y * s, a.z * s, b.z * s, a.w * s, b.w * s};
  unsigned w1[4], w2[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const __half ha = __float2half_rn(f[2 * j]), hb = __float2half_rn(f[2 * j + 1]);
    const __half la = __float2half_rn(f[2 * j] - __half2float(ha)), lb = __float2half_rn(f[2 * j + 1] - __half2float(hb));
    w1[j] = (unsigned)__half_as_ushort(ha) | ((unsigned)__half_as_ushort(hb) << 16);
    w2[j] = (unsigned)__half_as_ushort(la) | ((unsigned)__half_as_ushort(lb) << 16);
  }
  hi = make_uint4(w1[0], w1[1], w1[2], w1[3]);
  lo = make_uint4(w2[0], w2[1], w2[2], w2[3]);
}

#endif  // __CUDACC__

}  // namespace tlb
