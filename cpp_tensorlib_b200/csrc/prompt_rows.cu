// Row operations between the products of the int4 decoder's prompt pass, each one pass over its rows:
//
//   norm_split     x (+ b) -> residual, its RMS norm, the norm's fp16 planes for the next product
//   swiglu_split   gate | up rows -> silu(gate) * up, its planes
//   qkv_rows       q, k, v of a token: biases, rotation; q in place, k and v into the caches
//
// They do the work of add_rmsnorm / swiglu / split_heads / rope / kv_fill (fused_ops.cu, attn_prefill.cu) and
// split_f16_kernel with the same arithmetic, and the attention reads and writes token-major rows, so no
// head-major copy exists.  All are bound by memory: a row is read once, kept in shared memory for the row's
// sum or maximum, and written once.  Five launches a layer where there were fourteen: 143 us less a layer of 1000
// tokens at 3584 / 18944 columns, 32 us less a layer of 517 tokens at 896 / 4864.
#include <cuda_bf16.h>

#include "q4_planes.cuh"

namespace tlb {

namespace {

constexpr int SS_THREADS = 512;

// op over the block; the same value in every thread
template <class Op>
__device__ __forceinline__ float block_reduce(float v, float* sm, Op op, float (*in_warp)(float)) {
  v = in_warp(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sm[0];
  for (int w = 1; w < (int)((blockDim.x + 31) >> 5); w++) r = op(r, sm[w]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ float sum_in_warp(float v) { return warp_sum(v); }
__device__ __forceinline__ float max_in_warp(float v) { return warp_max(v); }
__device__ __forceinline__ float block_sum(float v, float* sm) {
  return block_reduce(v, sm, [](float a, float b) { return a + b; }, sum_in_warp);
}
__device__ __forceinline__ float block_max(float v, float* sm) {
  return block_reduce(v, sm, [](float a, float b) { return fmaxf(a, b); }, max_in_warp);
}

// the row in shared memory, whose largest magnitude is mx, as planes
__device__ __forceinline__ void store_planes(const float* row, int n, float mx, const Q4Planes& p) {
  const int e = q4_row_exponent(mx);
  const float s = ldexpf(1.0f, -e);
  if (threadIdx.x == 0) p.rowscale[blockIdx.x] = ldexpf(1.0f, e);
  uint4* hi = (uint4*)(p.hi + (size_t)blockIdx.x * n);
  uint4* lo = (uint4*)(p.lo + (size_t)blockIdx.x * n);
  for (int i = threadIdx.x; i < n / 8; i += blockDim.x) {
    uint4 a, b;
    q4_split8(((const float4*)row)[2 * i], ((const float4*)row)[2 * i + 1], s, a, b);
    hi[i] = a;
    lo[i] = b;
  }
}

// b NULL: the norm of x alone, and xout is not written
__global__ void norm_split_kernel(const float* x, const float* __restrict__ b, const float* __restrict__ w, float* xout,
                                  int n, float eps, Q4Planes p) {
  extern __shared__ float4 row4[];
  __shared__ float sm[32];
  float* row = (float*)row4;
  pdl_wait();
  pdl_launch_dependents();
  const size_t base = (size_t)blockIdx.x * n;
  float acc = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    float v = x[base + i];
    if (b) {
      v += b[base + i];
      xout[base + i] = v;
    }
    row[i] = v;
    acc += v * v;
  }
  const float inv = 1.0f / sqrtf(block_sum(acc, sm) / (float)n + eps);
  float mx = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = row[i] * inv * w[i];
    row[i] = v;
    mx = fmaxf(mx, fabsf(v));
  }
  store_planes(row, n, block_max(mx, sm), p);
}

__global__ void __launch_bounds__(SS_THREADS) swiglu_split_kernel(const float* __restrict__ gu, int ff, Q4Planes p) {
  extern __shared__ float4 row4[];
  __shared__ float sm[32];
  pdl_wait();
  pdl_launch_dependents();
  const float4* g4 = (const float4*)(gu + (size_t)blockIdx.x * 2 * ff);
  const float4* u4 = g4 + ff / 4;
  float mx = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < ff / 4; i += SS_THREADS) {
    const float4 g = __ldg(g4 + i), u = __ldg(u4 + i);
    const float4 m = make_float4((g.x / (1.0f + expf(-g.x))) * u.x, (g.y / (1.0f + expf(-g.y))) * u.y,
                                 (g.z / (1.0f + expf(-g.z))) * u.z, (g.w / (1.0f + expf(-g.w))) * u.w);
    row4[i] = m;
    mx = fmaxf(fmaxf(mx, fmaxf(fabsf(m.x), fabsf(m.y))), fmaxf(fabsf(m.z), fabsf(m.w)));
  }
  store_planes((const float*)row4, ff, block_max(mx, sm), p);
}

// One block per token.  The angles are those of rope_kernel (formed in double), once a token instead of once a
// head and token.
__global__ void qkv_rows_kernel(float* qkv, const float* __restrict__ bq, const float* __restrict__ bk,
                                const float* __restrict__ bv, void* __restrict__ Kc, void* __restrict__ Vc, int n_q,
                                int n_kv, int D, unsigned pos0, long long kv_stride, float base, int bf) {
  __shared__ float2 cs[64];
  const int half = D >> 1;
  const unsigned pos = pos0 + blockIdx.x;
  if ((int)threadIdx.x < half) {
    const double theta = exp2(-2.0 * (double)threadIdx.x / (double)D * log2((double)base));
    double sd, cd;
    sincos((double)pos * theta, &sd, &cd);
    cs[threadIdx.x] = make_float2((float)cd, (float)sd);
  }
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  float* row = qkv + (size_t)blockIdx.x * (n_q + 2 * n_kv) * D;
  const size_t slot = (size_t)pos * D;
  for (int i = threadIdx.x; i < (n_q + 2 * n_kv) * half; i += blockDim.x) {
    const int h = i / half, j = i - h * half;
    float x0 = row[h * D + j], x1 = row[h * D + j + half];
    const bool is_v = h >= n_q + n_kv;
    const int kh = h - n_q - (is_v ? n_kv : 0);
    const float* bias = h < n_q ? bq : (is_v ? bv : bk);
    if (bias) {
      const float* bp = bias + (h < n_q ? h : kh) * D;
      x0 += bp[j];
      x1 += bp[j + half];
    }
    if (!is_v) {
      const float2 r = cs[j];
      const float a = x0 * r.x - x1 * r.y;
      x1 = x0 * r.y + x1 * r.x;
      x0 = a;
    }
    if (h < n_q) {
      row[h * D + j] = x0;
      row[h * D + j + half] = x1;
      continue;
    }
    void* cache = is_v ? Vc : Kc;
    const size_t dst = (size_t)kh * kv_stride + slot + j;
    if (bf) {
      ((__nv_bfloat16*)cache)[dst] = __float2bfloat16_rn(x0);
      ((__nv_bfloat16*)cache)[dst + half] = __float2bfloat16_rn(x1);
    } else {
      ((float*)cache)[dst] = x0;
      ((float*)cache)[dst + half] = x1;
    }
  }
}

}  // namespace

// Widths whose row fits shared memory (192 of 227 KB) beside what the kernels declare themselves, in whole
// 16-byte pieces; other widths take the single operations.
bool prompt_rows_eligible(int n) { return n % 8 == 0 && n <= 49152; }

int launch_norm_split(const float* x, const float* b, const float* w, float* xout, int n, float eps, int rows,
                      const Q4Planes& p, cudaStream_t s) {
  // the thread count of launch_add_rmsnorm: the same partial sums
  int threads = ((n + 3) / 4 + 31) & ~31;
  threads = threads < 64 ? 64 : (threads > 1024 ? 1024 : threads);
  static std::atomic<unsigned long long> done{0};
  const int rc = ensure_dynamic_smem(norm_split_kernel, 49152 * 4, done);
  if (rc) return rc;
  LaunchCfg lc(dim3(rows), dim3(threads), (size_t)n * 4, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, norm_split_kernel, x, b, w, xout, n, eps, p));
  return TLB_OK;
}
int launch_swiglu_planes(const float* gu, int ff, int rows, const Q4Planes& p, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  const int rc = ensure_dynamic_smem(swiglu_split_kernel, 49152 * 4, done);
  if (rc) return rc;
  LaunchCfg lc(dim3(rows), dim3(SS_THREADS), (size_t)ff * 4, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, swiglu_split_kernel, gu, ff, p));
  return TLB_OK;
}
int launch_qkv_rows(float* qkv, const float* bq, const float* bk, const float* bv, void* Kc, void* Vc, int rows,
                    int n_q, int n_kv, int D, int pos0, long long kv_max, float base, int bf, cudaStream_t s) {
  LaunchCfg lc(dim3(rows), dim3(256), 0, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, qkv_rows_kernel, qkv, bq, bk, bv, Kc, Vc, n_q, n_kv, D, (unsigned)pos0, kv_max * D,
                              base, bf));
  return TLB_OK;
}

}  // namespace tlb
