// Causal attention over a prompt chunk against a bf16 cache on the tensor pipe (D = 64 or 128): the contract of
// cuda::attn_prefill / tl_attn_prefill_tiled_* with kv_bf16 (include/cuda.h:1171-1201,
// kernels/tensorlib_cuda.cu:1211-1350).  K, V [n_kv, kv_max, D] bf16; query p sits at absolute position
// pos0 + p and attends keys 0..pos0+p; q and out f32 rows with strides of their own.
//
//  * K and V are exact as operands of mma.sync.m16n8k16 bf16.  Queries (scaled by scale * log2 e) and weights are
//    f32 and enter as three bf16 planes each (8 + 8 + 8 mantissa bits, nothing dropped), so the products are those
//    of the f32 path: three MMAs a step where the tf32 split of attn_prefill_mma.cu would take two of half the
//    depth at half the rate, and no conversion of K or V.
//  * grid = (q heads, query tiles of 64), the tiles with most keys first over all heads.  Four warps own 16 query rows each, query
//    planes and output accumulators in registers; K/V tiles of 64 keys arrive by TMA (boxes of 64 keys x 64
//    dimensions, 128-byte swizzle) in a ring of three, 96 KB, so that two CTAs share an SM and the softmax of one
//    runs under the MMAs of the other.
//  * What bounds it is mma.sync: 6 D MACs a (query, key) pair, the tensor pipe busy for 61 % of an SM's active time;
//    the other side is the softmax and the latency between the two.  1000 queries x 28 heads of 128 took 551 us
//    on the CUDA cores, one f32 FMA a MAC; 114 us here head by head, 84 with the longest tiles first, 83 with the parameters
//    read in place.  At D = 128 a thread has 255 registers and spills 200 bytes.
//  * The last tile's rows past the chunk are cleared in shared memory (their weight is zero, but 0 * NaN is NaN).
//    Rows that come out NaN are computed again in plain f32 (attn_row_again), where infinite keys and values give what they
//    give on the CUDA cores.
#include "attn_common.cuh"
#include "rows_mma.cuh"

namespace tlb {

namespace {

constexpr int PB_QT = 64, PB_TK = 64, PB_THREADS = 128, PB_STAGES = 3;
constexpr int PB_BOX = 64 * 128;   // 64 keys x 64 bf16

template <int D>
struct PbCfg {
  static constexpr int SEGS = D / 64;
  static constexpr int TILE = 2 * SEGS * PB_BOX;   // K boxes, then V boxes
  static constexpr size_t BARS = (size_t)PB_STAGES * TILE;
  static constexpr size_t TOTAL = 1024 + BARS + PB_STAGES * 8;
};

struct PbParams {
  const float* q;
  const __nv_bfloat16 *K, *V;
  float* out;
  long long q_row, q_head, o_row, o_head;   // strides in floats
  int T, group, kv_rows, pos0;
  float scale;
  int* status;
};

// two f32 values as three bf16 planes
__device__ __forceinline__ void pb_split(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  hi = *(const uint32_t*)&h;
  rc_split(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u), mid, lo);
}
__device__ __forceinline__ void pb_ldm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void pb_ldmt(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// Four column tiles of one step, added to d in f32.  The three planes meet in an accumulator that starts at zero,
// the smallest first: an MMA cuts its sum to 24 bits without rounding, and a chain of them over a row's keys
// drifts (1.3e-6 of the result at 1000 keys, where f32 FMAs show 3.3e-7).
__device__ __forceinline__ void pb_step(float (*d)[4], const uint32_t (&lo)[4], const uint32_t (&mid)[4],
                                        const uint32_t (&hi)[4], const uint32_t (&b)[2][4]) {
  float t[4][4];
#pragma unroll
  for (int n = 0; n < 4; n++) t[n][0] = t[n][1] = t[n][2] = t[n][3] = 0.f;
#pragma unroll
  for (int n = 0; n < 4; n++) rc_mma(t[n], lo, b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
  for (int n = 0; n < 4; n++) rc_mma(t[n], mid, b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
  for (int n = 0; n < 4; n++) rc_mma(t[n], hi, b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
  for (int n = 0; n < 4; n++)
#pragma unroll
    for (int e = 0; e < 4; e++) d[n][e] += t[n][e];
}
__device__ __forceinline__ float pb_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// rows of the warp that came out NaN, again
template <int D>
__device__ __noinline__ void pb_again(const PbParams& p, unsigned a, unsigned b) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.x;
  const size_t kv = (size_t)(h / p.group) * p.kv_rows * D;
  for (int r = 0; r < 16; r++) {
    if (!(((r < 8 ? a : b) >> (4 * (r & 7))) & 15u)) continue;
    const int row = (int)(gridDim.y - 1 - blockIdx.y) * PB_QT + 16 * warp + r;
    const AttnRow<D> x = attn_row_again<D>(p.q + h * p.q_head + row * p.q_row, p.K + kv, p.V + kv,
                                           p.scale * 1.4426950408889634f, 0, p.pos0 + row + 1, 1);
    float* out = p.out + h * p.o_head + row * p.o_row + lane * (D / 32);
#pragma unroll
    for (int i = 0; i < D / 32; i++) out[i] = x.acc[i] / x.l;
  }
}

template <int D>
__global__ void __launch_bounds__(PB_THREADS, 2)
    attn_prefill_bf16_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                             const __grid_constant__ PbParams p) {
  using C = PbCfg<D>;
  constexpr int SEGS = C::SEGS, KS = D / 16, NT = D / 8;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = (uint64_t*)(base + C::BARS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int h = blockIdx.x, row0 = (h / p.group) * p.kv_rows;
  const int q0 = (int)(gridDim.y - 1 - blockIdx.y) * PB_QT;
  if (tid == 0) {
    for (int s = 0; s < PB_STAGES; s++) mbar_init(&full[s], 1);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();

  const int last_q = q0 + PB_QT < p.T ? q0 + PB_QT - 1 : p.T - 1;
  const int n_keys = p.pos0 + last_q + 1, n_tiles = (n_keys + PB_TK - 1) / PB_TK;
  auto issue = [&](int i) {
    const int s = i % PB_STAGES;
    unsigned char* dst = base + (size_t)s * C::TILE;
    mbar_expect_tx(&full[s], C::TILE);
#pragma unroll
    for (int sg = 0; sg < SEGS; sg++) {
      tma_load_2d(dst + sg * PB_BOX, &tmK, sg * 64, row0 + i * PB_TK, &full[s]);
      tma_load_2d(dst + (SEGS + sg) * PB_BOX, &tmV, sg * 64, row0 + i * PB_TK, &full[s]);
    }
  };
  if (tid == 0)
    for (int i = 0; i < PB_STAGES && i < n_tiles; i++) issue(i);

  const int ra = q0 + 16 * warp + g, rb = ra + 8;   // the lane's two query rows
  uint32_t qf[3][KS][4];
  {
    const float qs = p.scale * 1.4426950408889634f;
    const bool oka = ra < p.T, okb = rb < p.T;
    const float* qa = p.q + h * p.q_head + (oka ? ra : 0) * p.q_row + 2 * t;
    const float* qb = p.q + h * p.q_head + (okb ? rb : 0) * p.q_row + 2 * t;
#pragma unroll
    for (int k = 0; k < KS; k++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool ok = i & 1 ? okb : oka;
        float2 v = *(const float2*)((i & 1 ? qb : qa) + 16 * k + 8 * (i >> 1));
        if (!ok) v = make_float2(0.f, 0.f);
        pb_split(v.x * qs, v.y * qs, qf[0][k][i], qf[1][k][i], qf[2][k][i]);
      }
  }
  const int pa = p.pos0 + ra, pb = pa + 8;          // their positions
  const int first = p.pos0 + q0 + 16 * warp;        // the warp's first row's
  const bool works = q0 + 16 * warp < p.T;
  const int lim = first + 15 < n_keys - 1 ? first + 15 : n_keys - 1;
  // lane parts of the fragment addresses: row * 128 and the 16-byte chunk, swizzled by row & 7
  const uint32_t kr = (uint32_t)((lane & 7) + ((lane >> 4) << 3)) * 128u, kc = (uint32_t)((lane >> 3) & 1), sw = (uint32_t)(lane & 7);
  const uint32_t vr = (uint32_t)(lane & 15) * 128u, vc = (uint32_t)(lane >> 4);
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;

  bool dead = false;   // a bounded wait gave up: stop computing, but keep every rendezvous
  for (int it = 0; it < n_tiles; it++) {
    const int s_ = it % PB_STAGES, k0 = it * PB_TK;
    if (!dead && !mbar_wait_warp(&full[s_], (it / PB_STAGES) & 1, p.status, 720 + s_)) dead = true;
    unsigned char* tile = base + (size_t)s_ * C::TILE;
    if (n_keys - k0 < PB_TK) {   // the last tile only: values of rows past the chunk
      const int r0 = n_keys - k0, n = (PB_TK - r0) * 8;
      for (int i = tid; i < n * SEGS; i += PB_THREADS) {
        const int sg = i / n, j = i - sg * n;
        *(uint4*)(tile + (SEGS + sg) * PB_BOX + (r0 + (j >> 3)) * 128 + (j & 7) * 16) = make_uint4(0, 0, 0, 0);
      }
      __syncthreads();
    }
    if (!dead && works && k0 <= lim) {
      const uint32_t kt = smem_u32(tile), vt = kt + SEGS * PB_BOX;
      float s[8][4];
#pragma unroll
      for (int n = 0; n < 8; n++) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
      for (int k = 0; k < KS; k++) {
        const uint32_t a = kt + (uint32_t)(k >> 2) * PB_BOX + kr + ((((uint32_t)(k & 3) * 2 + kc) ^ sw) << 4);
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
          uint32_t b[2][4];
          pb_ldm(b[0], a + (2 * hf) * 2048u);
          pb_ldm(b[1], a + (2 * hf + 1) * 2048u);
          pb_step(s + 4 * hf, qf[2][k], qf[1][k], qf[0][k], b);
        }
      }
      if (k0 + PB_TK - 1 > first) {   // a tile the warp's first row does not see whole
#pragma unroll
        for (int n = 0; n < 8; n++) {
          const int key = k0 + 8 * n + 2 * t;
          if (key > pa) s[n][0] = -INFINITY;
          if (key + 1 > pa) s[n][1] = -INFINITY;
          if (key > pb) s[n][2] = -INFINITY;
          if (key + 1 > pb) s[n][3] = -INFINITY;
        }
      }
      float n0 = m0, n1 = m1;
#pragma unroll
      for (int n = 0; n < 8; n++) {
        n0 = fmaxf(n0, fmaxf(s[n][0], s[n][1]));
        n1 = fmaxf(n1, fmaxf(s[n][2], s[n][3]));
      }
#pragma unroll
      for (int x = 1; x < 4; x <<= 1) {
        n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, x));
        n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, x));
      }
      // a row whose scores are all -inf so far: 0 as the reference point, so that nothing becomes NaN
      const float r0 = n0 == -INFINITY ? 0.f : n0, r1 = n1 == -INFINITY ? 0.f : n1;
      const float f0 = pb_ex2(m0 - r0), f1 = pb_ex2(m1 - r1);
      m0 = n0;
      m1 = n1;
      l0 *= f0;
      l1 *= f1;
#pragma unroll
      for (int j = 0; j < NT; j++) {
        o[j][0] *= f0; o[j][1] *= f0;
        o[j][2] *= f1; o[j][3] *= f1;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {   // 16 keys a step
        uint32_t w[3][4];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          float* c = s[2 * k + e];
          c[0] = pb_ex2(c[0] - r0); c[1] = pb_ex2(c[1] - r0);
          c[2] = pb_ex2(c[2] - r1); c[3] = pb_ex2(c[3] - r1);
          l0 += c[0] + c[1];
          l1 += c[2] + c[3];
          pb_split(c[0], c[1], w[0][2 * e], w[1][2 * e], w[2][2 * e]);
          pb_split(c[2], c[3], w[0][2 * e + 1], w[1][2 * e + 1], w[2][2 * e + 1]);
        }
#pragma unroll
        for (int sg = 0; sg < SEGS; sg++) {
          const uint32_t a = vt + (uint32_t)sg * PB_BOX + (uint32_t)k * 2048u + vr;
#pragma unroll
          for (int hf = 0; hf < 2; hf++) {
            uint32_t b[2][4];
            pb_ldmt(b[0], a + ((((uint32_t)(2 * hf) * 2 + vc) ^ sw) << 4));
            pb_ldmt(b[1], a + ((((uint32_t)(2 * hf + 1) * 2 + vc) ^ sw) << 4));
            pb_step(o + 8 * sg + 4 * hf, w[2], w[1], w[0], b);
          }
        }
      }
    }
    __syncthreads();
    if (tid == 0 && it + PB_STAGES < n_tiles) issue(it + PB_STAGES);
  }

#pragma unroll
  for (int x = 1; x < 4; x <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, x);
    l1 += __shfl_xor_sync(0xffffffffu, l1, x);
  }
  const float i0 = 1.0f / l0, i1 = 1.0f / l1;
  float* oa = p.out + h * p.o_head + ra * p.o_row + 2 * t;
  bool nan_a = false, nan_b = false;
#pragma unroll
  for (int j = 0; j < NT; j++) {
    const float2 a = make_float2(o[j][0] * i0, o[j][1] * i0), b = make_float2(o[j][2] * i1, o[j][3] * i1);
    nan_a |= a.x != a.x || a.y != a.y;
    nan_b |= b.x != b.x || b.y != b.y;
    if (ra < p.T) *(float2*)(oa + 8 * j) = a;
    if (rb < p.T) *(float2*)(oa + 8 * p.o_row + 8 * j) = b;
  }
  const unsigned again_a = __ballot_sync(0xffffffffu, nan_a && ra < p.T), again_b = __ballot_sync(0xffffffffu, nan_b && rb < p.T);
  if (again_a | again_b) pb_again<D>(p, again_a, again_b);
}

template <int D>
int pb_launch(const PbParams& p, const void* K, const void* V, int n_q, int n_kv, cudaStream_t stream) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return set_error(TLB_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
  CUtensorMap tm[2];
  cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)n_kv * (cuuint64_t)p.kv_rows};
  cuuint64_t strides[1] = {(cuuint64_t)D * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)PB_TK};
  cuuint32_t es[2] = {1, 1};
  for (int i = 0; i < 2; i++) {
    CUresult r = enc(&tm[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(i ? V : K), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(TLB_ERR_CUDA, "attn_prefill: tensor map encode failed");
  }
  static std::atomic<unsigned long long> attr_done{0};
  const int rc = ensure_dynamic_smem(attn_prefill_bf16_kernel<D>, (int)PbCfg<D>::TOTAL, attr_done);
  if (rc) return rc;
  LaunchCfg lc(dim3(n_q, (p.T + PB_QT - 1) / PB_QT), dim3(PB_THREADS), PbCfg<D>::TOTAL, stream, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, attn_prefill_bf16_kernel<D>, tm[0], tm[1], p));
  return TLB_OK;
}

}  // namespace

int attn_prefill_bf16_launch(DeviceCtx* c, const float* q, long long q_row, long long q_head, const void* K,
                             const void* V, float* out, long long o_row, long long o_head, int n_q, int n_kv, int T,
                             long long kv_max, int D, float scale, int pos0, cudaStream_t s) {
  // tile coordinates are ints; so many rows of a bf16 cache are more than a GPU holds
  if ((long long)n_kv * kv_max >= (1ll << 31) - PB_TK)
    return set_error(TLB_ERR_UNSUPPORTED, "attn_prefill: a bf16 cache of 2^31 rows or more");
  PbParams p;
  p.q = q; p.q_row = q_row; p.q_head = q_head;
  p.K = (const __nv_bfloat16*)K; p.V = (const __nv_bfloat16*)V;
  p.out = out; p.o_row = o_row; p.o_head = o_head;
  p.T = T; p.group = n_q / n_kv; p.kv_rows = (int)kv_max; p.pos0 = pos0;
  p.scale = scale; p.status = c->status;
  return D == 128 ? pb_launch<128>(p, K, V, n_q, n_kv, s) : pb_launch<64>(p, K, V, n_q, n_kv, s);
}

}  // namespace tlb
