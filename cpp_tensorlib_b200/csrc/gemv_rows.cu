// One-row matrix product of the layer-stack decoder, y = W . f(x), with its neighbours fused: on the
// staged activation in front, the residual sum that a norm of the preceding sublayer's output ends in,
// an RMS norm (whole row, or a segment in equal parts) and a silu gate; a residual add, the clipped
// gated unit or the square of relu behind.  W is bf16 or f32 row-major, everything else f32.
//
// HBM bound in the long run, but a token's launch streams 17 - 46 MB (2.6 - 7 us) and used to take 4 us beyond that: what
// it costs is the chain from the end of the launch in front to the first weight used.  So
//   - a block takes at most half an SM (112 KB, 96 registers x 288 threads): the next launch's block fits beside it and has
//     its ring of weights full when this launch ends.  One block an SM, a contiguous range of rows each, so that a stage
//     of the ring (8 rows of 2048, 4 of 4096, ...) is one bulk copy.  (Rows of 16 - 32 KB, up to
//     eight chunks a thread, take the registers of a whole SM: the next launch's ring starts when a block ends);
//   - a thread owns the same 16-byte chunks of every row: its activations go from memory to its registers, without shared
//     memory or a barrier, all loads in flight at once;
//   - the factor of a norm over the whole row multiplies the sums instead of the activations; the norms' weights are
//     fetched in front of the wait; the sums of several rows go through the warp together;
//   - the sums of a norm in parts come from the chunks that the threads hold: a second look at the row waited 1 - 2 us behind
//     the weights of the next launch (a token of the 8-layer Mamba stack 305 -> 285 us, of the latent stack 386 -> 377).
// Launches of one shape behind each other, cold weights, us (before: two rows a warp in registers, two blocks an SM):
//   2048 -> 10304 with norm 11.1 -> 10.1, 2048 -> 11264 11.7 -> 10.8, 4096 -> 2048 6.9 -> 4.9, 5632 -> 2048 7.3 -> 7.0;
//   the first with the weights in the L2 already: 11.0 -> 7.1.
// What is left is the HBM idling from a launch's last bulk copy to the next one's first free stage, about 3 us.  Tried
// without gain: the weights behind the ring brought to the L2 early by prefetches (they fetch into the far half of the
// L2: a read behind them runs at 31 bytes a clock and SM, behind a load at 70) or by loads of a word a line (they delay
// the activations of the launch that still runs); stages of half the size (305 -> 330 us a token of the 8-layer stack).
// Weights are marked evict-first in the L2: a token streams gigabytes of them once, and what every launch needs again --
// instructions, states, activations -- should stay.
#include "mixers.cuh"

namespace tlb {

namespace {

constexpr int RG_WARPS = 8, RG_THREADS = RG_WARPS * 32;   // and a warp that only requests weights
// Shared memory of a block: at most half an SM's, so that the next launch's blocks fit beside this one's.
constexpr size_t RG_SMEM_SHARED = 112 * 1024, RG_SMEM_MAX = 226 * 1024;

struct RowPlan {
  int stages, stage_rows, rows_max;   // ring; rows of a stage; most rows of a block
  int wpr;                            // warps on a row
  int part_chunks;                    // 16-byte chunks' worth of elements of a norm's part
  unsigned part_magic;                // ceil(2^32 / part_chunks), 0 for one: a chunk's part without a division
  int* status;
};

// base[i .. i + N) where it lies in [0, n), else 0: N and n multiples of N, 16-byte aligned
template <int N>
__device__ __forceinline__ void rg_ld(const float* base, int i, int n, float (&o)[N]) {
  const bool on = i >= 0 && i < n;
  const float4* at = (const float4*)(base + (on ? i : 0));
#pragma unroll
  for (int k = 0; k < N; k += 4) {
    const float4 v = __ldcg(at + k / 4);
    o[k] = on ? v.x : 0.f; o[k + 1] = on ? v.y : 0.f; o[k + 2] = on ? v.z : 0.f; o[k + 3] = on ? v.w : 0.f;
  }
}

// A norm over the whole row: its factor multiplies the row sums instead of the elements.  (Of a segment, in parts or not,
// the elements are multiplied with their part's factor, gs.)
__device__ __forceinline__ bool rg_whole(const RowGemv& p) { return p.nw && p.n_groups == 1 && p.n_len == p.K; }
// N elements of the staged row from e0 on: v holds them as they are in x, w the norm's weights, r and rn the residual and
// its weights, g the gate; s is the residual's scale
// (the row, the segment and its parts are whole pieces of N elements)
template <int N>
__device__ __forceinline__ void rg_prepare(const RowGemv& p, int e0, float (&v)[N], const float (&w)[N], const float (&r)[N],
                                           const float (&rn)[N], const float (&g)[N], float s, const float* gs, unsigned magic, float& sq) {
  if (p.res) {
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = fmaf(v[k] * s, rn[k], r[k]);
    if (p.xout && blockIdx.x == 0) {
      if (e0 < p.K)
#pragma unroll
        for (int k = 0; k < N; k += 4) *(float4*)(p.xout + e0 + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    }
  }
#pragma unroll
  for (int k = 0; k < N; k++) sq = fmaf(v[k], v[k], sq);
  if (!p.nw) return;
  if (rg_whole(p)) {
#pragma unroll
    for (int k = 0; k < N; k++) v[k] *= p.gate ? w[k] * silu_f(g[k]) : w[k];
    return;
  }
  if (e0 + N <= p.n_off || e0 >= p.n_off + p.n_len) return;
  const unsigned c = (unsigned)((e0 - p.n_off) / N);
  const float f = gs[magic ? __umulhi(c, magic) : c];
#pragma unroll
  for (int k = 0; k < N; k++) v[k] *= p.gate ? f * w[k] * silu_f(g[k]) : f * w[k];
}
// R sums over a warp: afterwards lane l holds the sum of v[rg_sum_of<R>(l)] in v[0]
template <int R>
__device__ __forceinline__ int rg_sum_of(int lane) { return R == 1 ? 0 : (lane >> 4) + (R >= 4 ? ((lane >> 3) & 1) * 2 : 0) + (R >= 8 ? ((lane >> 2) & 1) * 4 : 0); }
template <int R>
__device__ __forceinline__ void rg_warp_sums(float (&v)[R], int lane) {
  int o = 16;
#pragma unroll
  for (int n = R; n > 1; n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; i++) {
      const float send = up ? v[2 * i] : v[2 * i + 1], keep = up ? v[2 * i + 1] : v[2 * i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    o >>= 1;
  }
#pragma unroll
  for (int k = 0; k < 5; k++)
    if ((16 >> k) <= o) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16 >> k);
}
// sums of the eight warps, the same in every thread behind a barrier
__device__ __forceinline__ float rg_total(const float* red) {
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < RG_WARPS; w++) t += red[w];
  return t;
}
__device__ __forceinline__ void rg_sync() { asm volatile("bar.sync 1, %0;" ::"n"(RG_THREADS) : "memory"); }
__device__ __forceinline__ void rg_emit(const RowGemv& p, int n, float a, float b, float y0) {
  if (p.epi == 2) p.y[n >> 1] = glu_clipped(a, b, p.limit);
  else p.y[n] = p.epi == 1 ? y0 + a : (p.epi == 3 ? relu2(a) : a);
}
__host__ __device__ constexpr int rg_rows_of(int jn) { return jn == 1 ? 8 : (jn == 2 ? 4 : (jn <= 4 ? 2 : 1)); }

// JN: 16-byte chunks of a row that a thread owns
template <typename WT, int JN>
__global__ void __launch_bounds__(RG_THREADS + 32, JN < 8 ? 2 : 1) row_gemv_kernel(const __grid_constant__ RowGemv p,
                                                                      const __grid_constant__ RowPlan pl) {
  constexpr int CE = Vec16<WT>::N, RB = rg_rows_of(JN);
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float red[2][RG_WARPS];
  __shared__ __align__(8) uint64_t full[16], empty[16];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, S = pl.stages;
  const int u = p.epi == 2 ? 2 : 1, units = (p.N + u - 1) / u, b = blockIdx.x;
  const int ub = units / (int)gridDim.x, ur = units - ub * (int)gridDim.x;
  const int r0 = (b * ub + (b < ur ? b : ur)) * u;
  int rows = (ub + (b < ur)) * u;
  if (rows > p.N - r0) rows = p.N - r0;
  const int RS = pl.stage_rows, nst = (rows + RS - 1) / RS, chunks = (int)(p.ldw / CE);
  const size_t row_bytes = (size_t)p.ldw * sizeof(WT), stage_bytes = RS * row_bytes;
  float* part = (float*)(smem + S * stage_bytes);   // [wpr][rows_max]
  auto request = [&](int i, int st, uint64_t pol) {
    const int n = rows - i * RS < RS ? rows - i * RS : RS;
    mbar_expect_tx(&full[st], (uint32_t)(n * row_bytes));
    bulk_load_1d_hint(smem + st * stage_bytes, (const unsigned char*)p.W + (size_t)r0 * row_bytes + i * stage_bytes,
                      (uint32_t)(n * row_bytes), &full[st], pol);
  };
  if (tid == RG_THREADS) {
    for (int i = 0; i < S; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], RG_WARPS); }
    mbar_fence_init();
    const uint64_t pol = l2_evict_first_policy();
    for (int i = 0; i < S && i < nst; i++) request(i, i, pol);
  }
  __syncthreads();
  if (warp == RG_WARPS) {
    if (lane) return;
    const uint64_t pol = l2_evict_first_policy();
    int st = 0;
    unsigned parity = 0;
    for (int i = S; i < nst; i++) {
      if (!mbar_wait_bounded(&empty[st], parity, pl.status, 801)) break;
      request(i, st, pol);
      if (++st == S) { st = 0; parity ^= 1u; }
    }
    return;
  }
  if (p.nw)   // the norms' weights into the L2
    for (int i = tid * 32; i < p.n_len; i += RG_THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.nw + i));
  if (p.rn)
    for (int i = tid * 32; i < p.K; i += RG_THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.rn + i));
  const int wpr = pl.wpr, G = RG_WARPS / wpr, grp = warp / wpr, wsub = warp - grp * wpr;
  const int c0 = JN == 1 ? wsub * 32 + lane : tid;   // this thread's chunks: c0, c0 + 256, ...
  // what fits the registers beside the row is fetched with it, the norms' weights in front of the wait
  constexpr bool FEW = JN <= 2, ONE = JN == 1;
  float x[JN][CE], nw[FEW ? JN : 1][CE], gate[FEW ? JN : 1][CE], rn[CE], res[CE];
  auto ld_nw = [&](int j, float (&o)[CE]) { if (p.nw) rg_ld<CE>(p.nw, (c0 + j * RG_THREADS) * CE - p.n_off, p.n_len, o); };
  auto ld_gate = [&](int j, float (&o)[CE]) { if (p.gate) rg_ld<CE>(p.gate, (c0 + j * RG_THREADS) * CE - p.n_off, p.n_len, o); };
  auto ld_rn = [&](int j) { if (p.rn) rg_ld<CE>(p.rn, (c0 + j * RG_THREADS) * CE, p.K, rn); };
  auto ld_res = [&](int j) { if (p.res) rg_ld<CE>(p.res, (c0 + j * RG_THREADS) * CE, p.K, res); };
  if (FEW)
#pragma unroll
    for (int j = 0; j < JN; j++) ld_nw(j, nw[FEW ? j : 0]);
  if (ONE) ld_rn(0);
  pdl_wait();
#pragma unroll
  for (int j = 0; j < JN; j++) rg_ld<CE>(p.x, (c0 + j * RG_THREADS) * CE, p.K, x[j]);
  if (ONE) ld_res(0);
  if (FEW)
#pragma unroll
    for (int j = 0; j < JN; j++) ld_gate(j, gate[FEW ? j : 0]);
  const float y0 = p.epi == 1 && tid < rows ? __ldcg(p.y + r0 + tid) : 0.f;   // what the row is added to
  pdl_launch_dependents();
  float s = 0.f, sq = 0.f;
  if (p.res) {   // 1 / rms of the preceding sublayer's output
#pragma unroll
    for (int i = 0; i < JN * CE; i++) sq = fmaf(x[i / CE][i % CE], x[i / CE][i % CE], sq);
    sq = warp_sum(grp == 0 ? sq : 0.f);
    if (lane == 0) red[0][warp] = sq;
    rg_sync();
    s = rsqrtf(rg_total(red[0]) / p.K + p.eps);
    sq = 0.f;
  }
  float* gs = part + pl.wpr * pl.rows_max;
  if (p.nw && !rg_whole(p)) {
    // the parts' sums from the chunks' (a part is whole chunks), a warp a part: no second look at the row, which would
    // wait behind the next launch's weights
    float* cs = gs + p.n_groups;
    const int lo = p.n_off / CE, m = pl.part_chunks;
#pragma unroll
    for (int j = 0; j < JN; j++) {
      const int c = c0 + j * RG_THREADS - lo;
      if (grp == 0 && c >= 0 && c < m * p.n_groups) {
        float q = 0.f;
#pragma unroll
        for (int e = 0; e < CE; e++) q = fmaf(x[j][e], x[j][e], q);
        cs[c] = q;
      }
    }
    rg_sync();
#pragma unroll 1
    for (int g = warp; g < p.n_groups; g += RG_WARPS) {
      float q = 0.f;
#pragma unroll 2
      for (int c = lane; c < m; c += 32) q += cs[g * m + c];
      q = warp_sum(q);
      if (lane == 0) gs[g] = rsqrtf(q / (m * CE) + p.eps) * p.nscale;
    }
    rg_sync();
  }
#pragma unroll
  for (int j = 0; j < JN; j++) {
    if (!ONE) { ld_rn(j); ld_res(j); }
    if (!FEW) { ld_nw(j, nw[0]); ld_gate(j, gate[0]); }
    rg_prepare<CE>(p, (c0 + j * RG_THREADS) * CE, x[j], nw[FEW ? j : 0], res, rn, gate[FEW ? j : 0], s, gs, pl.part_magic, sq);
  }
  if (rg_whole(p)) {
    sq = warp_sum(grp == 0 ? sq : 0.f);
    if (lane == 0) red[1][warp] = sq;
  }
  bool ok = true;
  int st = 0;
  unsigned parity = 0;
  // chunks that the row does not have: its first is read and dropped
  constexpr int SURE = JN < 8 ? JN - 1 : 4;
  auto has = [&](int j) { return j < SURE || c0 + j * RG_THREADS < chunks; };
  const uint32_t at = smem_u32(smem) + (uint32_t)(grp * row_bytes) + (uint32_t)c0 * 16u, rstep = (uint32_t)(G * row_bytes);
  const int row_of = rg_sum_of<RB>(lane) * G + grp;
  float* dst = part + wsub * pl.rows_max;
  for (int i = 0; i < nst; i++) {
    ok = ok && mbar_poll_warp(&full[st], parity, pl.status, 800);
    const uint32_t base = at + (uint32_t)(st * stage_bytes);
    float acc[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) {   // (rows behind the last one: whatever the slot held, and not kept)
      acc[r] = 0.f;
#pragma unroll
      for (int j = 0; j < JN; j++) {
        uint4 w;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                     : "r"(base + r * rstep + (has(j) ? (uint32_t)j * (RG_THREADS * 16u) : 0u - (uint32_t)c0 * 16u)));
        if (!has(j)) w = make_uint4(0, 0, 0, 0);
        float f[CE];
        widen16(w, f, (const WT*)nullptr);
#pragma unroll
        for (int e = 0; e < CE; e++) acc[r] = fmaf(f[e], x[j][e], acc[r]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
    if (++st == S) { st = 0; parity ^= 1u; }
    rg_warp_sums<RB>(acc, lane);
    const int row = i * RS + row_of;
    if ((lane & (32 / RB - 1)) == 0 && row < rows) dst[row] = acc[0];
  }
  rg_sync();
  const float f = rg_whole(p) ? rsqrtf(rg_total(red[1]) / p.K + p.eps) * p.nscale : 1.f;
  auto row_sum = [&](int r) {
    float q[RG_WARPS], a = 0.f;
#pragma unroll
    for (int k = 0; k < RG_WARPS; k++) q[k] = k < wpr ? part[k * pl.rows_max + r] : 0.f;
#pragma unroll
    for (int k = 0; k < RG_WARPS; k++) a += q[k];
    return a * f;
  };
  for (int r = tid * u; r < rows; r += RG_THREADS * u)
    rg_emit(p, r0 + r, row_sum(r), u == 2 ? row_sum(r + 1) : 0.f, p.epi != 1 || r == tid ? y0 : p.y[r0 + r]);
}

// ---- rows too long for the registers of a block, and rows of odd widths or places ------------
// The staged row in shared memory, weights straight from memory: a stream of ks adjacent warps owns one row, or two adjacent
// rows (gate and up interleaved), each warp its own part of K; ks is picked on the host so that the streams of all SMs come
// out even.  Every warp keeps eight 16-byte loads in flight plus the next eight, and the first eight are issued in front of
// the wait.
// What lies where, us a token of models with such products, streams / ring: rows of 16384 in bf16 (`down` of four layers of
// 4096 x 16384) 460 / 436, of 14336 371 / 362, of 10240 282 / 275; f32 rows of 8192 281 / 285, of 4928 188 / 188.  Longer rows
// do not fit the ring's registers: 20000 in bf16 325 (a block for a row at a time, three barriers a row, 393), 16384 in f32
// 769 (951).
constexpr size_t RS_SMEM_MAX = 225 * 1024;

__device__ __forceinline__ uint4 rs_ld(const void* p, uint64_t pol) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(pol));
  return v;
}

// x into xs [ldw], zero behind K; returns this thread's share of its sum of squares.  Kept short: a
// launch runs this code once, from a cold instruction cache.
__device__ __forceinline__ float rs_stage(const RowGemv& p, float* xs) {
  float sq = 0.f;
  const int k4 = ((uintptr_t)p.x & 15) ? 0 : p.K / 4;   // rows of an odd width go one by one
  for (int i0 = threadIdx.x; i0 < k4; i0 += 4 * RG_THREADS) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * RG_THREADS < k4) v[u] = ((const float4*)p.x)[i0 + u * RG_THREADS];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * RG_THREADS < k4) {
        ((float4*)xs)[i0 + u * RG_THREADS] = v[u];
        sq = fmaf(v[u].x, v[u].x, fmaf(v[u].y, v[u].y, fmaf(v[u].z, v[u].z, fmaf(v[u].w, v[u].w, sq))));
      }
  }
#pragma unroll 1
  for (int i = 4 * k4 + threadIdx.x; i < p.ldw; i += RG_THREADS) {
    const float x = i < p.K ? p.x[i] : 0.f;
    xs[i] = x;
    sq = fmaf(x, x, sq);
  }
  return sq;
}

// the preceding sublayer's output, normed, added to the residual: every block computes the row, block 0
// leaves it for the launches behind.  Returns the thread's share of the new row's sum of squares.
__device__ __forceinline__ float rs_residual(const RowGemv& p, float* xs, float sq, float* red) {
  const float s = rsqrtf(block_sum(sq, red) / p.K + p.eps);
  sq = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < p.K; i += RG_THREADS) {
    const float v = fmaf(xs[i] * s, p.rn[i], p.res[i]);
    xs[i] = v;
    if (p.xout && blockIdx.x == 0) p.xout[i] = v;
    sq = fmaf(v, v, sq);
  }
  return sq;
}

// the norm in place: the whole row by the block, a segment in parts a warp each
__device__ __forceinline__ void rs_norm(const RowGemv& p, float* xs, float sq, float* red) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (p.n_groups == 1 && p.n_len == p.K) {
    const float s = rsqrtf(block_sum(sq, red) / p.K + p.eps) * p.nscale;
#pragma unroll 4
    for (int i = tid; i < p.K; i += RG_THREADS) xs[i] *= p.gate ? s * p.nw[i] * silu_f(p.gate[i]) : s * p.nw[i];
    return;
  }
  __syncthreads();
  const int m = p.n_len / p.n_groups;
#pragma unroll 1
  for (int g = tid >> 5; g < p.n_groups; g += RG_WARPS) {
    float* seg = xs + p.n_off + g * m;
    float q = 0.f;
#pragma unroll 4
    for (int i = lane; i < m; i += 32) q = fmaf(seg[i], seg[i], q);
    const float s = rsqrtf(warp_sum(q) / m + p.eps) * p.nscale;
#pragma unroll 4
    for (int i = lane; i < m; i += 32)
      seg[i] *= p.gate ? s * p.nw[g * m + i] * silu_f(p.gate[g * m + i]) : s * p.nw[g * m + i];
  }
}

template <int R>
__device__ __forceinline__ void rs_emit(const RowGemv& p, int rg, const float (&a)[R]) {
  if (p.epi == 2) {
    if (R == 2) rg_emit(p, 2 * rg, a[0], a[R - 1], 0.f);
    return;
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int n = rg * R + r;
    if (n < p.N) rg_emit(p, n, a[r], 0.f, p.epi == 1 ? p.y[n] : 0.f);
  }
}

template <typename WT, int R>
__global__ void __launch_bounds__(RG_THREADS, 2) row_gemv_stream_kernel(const __grid_constant__ RowGemv p, int ks) {
  constexpr int CE = Vec16<WT>::N, U = 8 / R;
  extern __shared__ __align__(16) float xs[];   // [ldw], then the streams' partial sums
  __shared__ float red[33];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int groups = (p.N + R - 1) / R, ns = RG_WARPS / ks, stream = warp / ks, sub = warp - stream * ks;
  const int stride = gridDim.x * ns, chunks = (int)(p.ldw / CE), per = (chunks + ks - 1) / ks;
  const int c_lo = sub * per, c_hi = c_lo + per < chunks ? c_lo + per : chunks;
  float* part = xs + p.ldw;                     // [local group][stream][R][ks]
  const WT* W = (const WT*)p.W;
  const uint64_t pol = l2_evict_first_policy();
  int rg = blockIdx.x * ns + stream, cb = c_lo, loc = 0;
  uint4 cur[R][U], nxt[R][U];
  auto fetch = [&](uint4 (&w)[R][U], int g, int b) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const WT* row = W + (size_t)(g * R + r < p.N ? g * R + r : p.N - 1) * p.ldw;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int c = b + lane + 32 * u;
        w[r][u] = c < c_hi ? rs_ld(row + (size_t)c * CE, pol) : make_uint4(0, 0, 0, 0);
      }
    }
  };
  if (rg < groups) fetch(cur, rg, cb);
  if (p.nw)   // the norm's weights into the L2
    for (int i = tid * 32; i < p.n_len; i += RG_THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.nw + i));
  if (p.rn)
    for (int i = tid * 32; i < p.K; i += RG_THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.rn + i));
  pdl_wait();
  pdl_launch_dependents();
  float sq = rs_stage(p, xs);
  if (p.res) sq = rs_residual(p, xs, sq, red);
  if (p.nw) rs_norm(p, xs, sq, red);
  __syncthreads();
  float acc[R][2];
#pragma unroll
  for (int r = 0; r < R; r++) acc[r][0] = acc[r][1] = 0.f;
  while (rg < groups) {
    int ng = rg, nb = cb + 32 * U;
    if (nb >= c_hi) { ng += stride; nb = c_lo; }
    if (ng < groups) fetch(nxt, ng, nb);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int c = cb + lane + 32 * u;
      if (c < c_hi) {
        float x[CE];
#pragma unroll
        for (int e = 0; e < CE; e += 4) {
          const float4 v = *(const float4*)(xs + (size_t)c * CE + e);
          x[e] = v.x; x[e + 1] = v.y; x[e + 2] = v.z; x[e + 3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
          float w[CE];
          widen16(cur[r][u], w, (const WT*)nullptr);
#pragma unroll
          for (int e = 0; e < CE; e++) acc[r][e & 1] = fmaf(w[e], x[e], acc[r][e & 1]);
        }
      }
    }
    if (ng != rg) {
      float a[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        a[r] = warp_sum(acc[r][0] + acc[r][1]);
        acc[r][0] = acc[r][1] = 0.f;
      }
      if (lane == 0) {
        if (ks == 1) {
          rs_emit<R>(p, rg, a);
        } else {
#pragma unroll
          for (int r = 0; r < R; r++) part[((loc * ns + stream) * R + r) * ks + sub] = a[r];
        }
      }
      loc++;
    }
    rg = ng;
    cb = nb;
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int u = 0; u < U; u++) cur[r][u] = nxt[r][u];
  }
  if (ks == 1) return;
  __syncthreads();
  for (int i = tid;; i += RG_THREADS) {
    const int l = i / ns, g = (blockIdx.x * ns + i - l * ns) + l * stride;
    if (l * stride + (int)blockIdx.x * ns >= groups) break;
    if (g >= groups) continue;
    float a[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      a[r] = 0.f;
      for (int k = 0; k < ks; k++) a[r] += part[(i * R + r) * ks + k];
    }
    rs_emit<R>(p, g, a);
  }
}

template <typename WT, int R>
int rs_launch(DeviceCtx* c, const RowGemv& p, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  const int rc = ensure_dynamic_smem(row_gemv_stream_kernel<WT, R>, RS_SMEM_MAX, done);
  if (rc) return rc;
  const int groups = (p.N + R - 1) / R, chunks = (int)(p.ldw / Vec16<WT>::N), full = 2 * c->sm_count;
  // warps a stream (single rows): the fewest that come within 3 % of the most even division
  int ks = 1;
  double best = 1e30;
  for (int k = 1; k <= RG_WARPS; k *= 2) {
    if (k > 1 && chunks / k < 32 * 4) break;
    const int ns = RG_WARPS / k;
    const double cost = (double)((groups + full * ns - 1) / (full * ns)) / k;
    if (cost < best * 0.97) { best = cost; ks = k; }
    if (R == 2) break;   // two rows a warp: the extra sums cost more than the unevenness
  }
  auto blocks = [&] {
    const int ns = RG_WARPS / ks, need = (groups + ns - 1) / ns;
    return need < full ? need : full;
  };
  auto bytes = [&] {   // the row and, of streams of several warps, their partial sums
    const int ns = RG_WARPS / ks, all = blocks() * ns, local = (groups + all - 1) / all;
    return ((size_t)p.ldw + (ks > 1 ? (size_t)local * ns * R * ks : 0)) * sizeof(float);
  };
  if (bytes() > RS_SMEM_MAX) ks = 1;
  const int ctas = blocks();
  const size_t smem = bytes();
  if (smem > RS_SMEM_MAX) return set_error(TLB_ERR_UNSUPPORTED, "row_gemv: the activation row does not fit the shared-memory stage");
  LaunchCfg lc(dim3(ctas), dim3(RG_THREADS), smem, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, row_gemv_stream_kernel<WT, R>, p, ks));
  return TLB_OK;
}

template <typename WT, int JN>
int rg_launch(const RowGemv& p, const RowPlan& pl, int ctas, size_t smem, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  const int rc = ensure_dynamic_smem(row_gemv_kernel<WT, JN>, RG_SMEM_MAX, done);
  if (rc) return rc;
  LaunchCfg lc(dim3(ctas), dim3(RG_THREADS + 32), smem, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, row_gemv_kernel<WT, JN>, p, pl));
  return TLB_OK;
}
template <typename WT>
int rg_plan_launch(DeviceCtx* c, const RowGemv& p, cudaStream_t s) {
  constexpr int CE = Vec16<WT>::N;
  const int chunks = (int)(p.ldw / CE), u = p.epi == 2 ? 2 : 1, units = (p.N + u - 1) / u;
  auto aligned = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
  const bool vec = aligned(p.x) && aligned(p.res) && aligned(p.rn) && aligned(p.nw) && aligned(p.gate) && aligned(p.xout) &&
                   p.K % CE == 0 &&
                   (!p.nw || (p.n_off % CE == 0 && p.n_len % CE == 0 && (p.n_len / p.n_groups) % CE == 0));
  const int groups = p.nw ? p.n_groups : 0;
  const int need = (chunks + RG_THREADS - 1) / RG_THREADS, jn = need <= 4 ? need : (need <= 8 ? 8 : 0);
  const int ctas = units < c->sm_count ? units : c->sm_count;
  RowPlan pl{};
  pl.status = c->status;
  pl.rows_max = (units + ctas - 1) / ctas * u;
  if (vec && p.nw) {
    pl.part_chunks = p.n_len / p.n_groups / CE;
    pl.part_magic = (unsigned)(((1ull << 32) + pl.part_chunks - 1) / pl.part_chunks);   // exact below 2^16 chunks; 1: 0
  }
  pl.wpr = RG_WARPS;
  while (pl.wpr > 1 && chunks <= pl.wpr / 2 * 32) pl.wpr /= 2;
  const size_t row = (size_t)p.ldw * sizeof(WT), tail = ((size_t)pl.wpr * pl.rows_max + groups + (groups ? p.n_len / CE : 0)) * sizeof(float) + 16;
  pl.stage_rows = jn ? rg_rows_of(jn) * (RG_WARPS / pl.wpr) : 1;
  const size_t stage = row * pl.stage_rows;
  const int nst = (pl.rows_max + pl.stage_rows - 1) / pl.stage_rows;
  pl.stages = nst < 16 ? nst : 16;
  while (pl.stages > 2 && pl.stages * stage + tail > RG_SMEM_SHARED) pl.stages--;
  const size_t smem = pl.stages * stage + tail;
  if (!jn || !vec || smem > RG_SMEM_MAX) {
    // two rows a stream where the rows come in pairs, or where there are enough of them to fill the SMs
    const bool two = p.epi == 2 || p.N >= 2 * 2 * c->sm_count * RG_WARPS;
    return two ? rs_launch<WT, 2>(c, p, s) : rs_launch<WT, 1>(c, p, s);
  }
  if (jn == 1) return rg_launch<WT, 1>(p, pl, ctas, smem, s);
  if (jn == 2) return rg_launch<WT, 2>(p, pl, ctas, smem, s);
  if (jn == 3) return rg_launch<WT, 3>(p, pl, ctas, smem, s);
  if (jn == 4) return rg_launch<WT, 4>(p, pl, ctas, smem, s);
  return rg_launch<WT, 8>(p, pl, ctas, smem, s);
}

// ---- row ops of the prompt pass --------------------------------------------------------------
template <typename OT>
__global__ void __launch_bounds__(256) rms_rows_kernel(const float* __restrict__ x, long long ldx,
                                                       const float* __restrict__ w, OT* __restrict__ out, long long ldo,
                                                       int n, float eps, float scale) {
  __shared__ float red[33];
  pdl_wait();
  pdl_launch_dependents();
  const float* row = x + (size_t)blockIdx.x * ldx;
  OT* dst = out + (size_t)blockIdx.x * ldo;
  float sq = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) sq = fmaf(row[i], row[i], sq);
  sq = block_sum(sq, red);
  const float r = rsqrtf(sq / n + eps) * scale;
  for (int i = threadIdx.x; i < n; i += 256) put(dst + i, row[i] * r * w[i]);
}

// Both of these with a row in a block's registers, 16 bytes an access and all of them in front of the sum: the kernels
// beside this one load in two rounds, 4 bytes an access.  RES: x += norm(v) * w, also to out; else out = norm(v) * w.
// HBM bound; 3001 rows of 2048 with the residual sum 22.5 -> 12.0 us (86 MB), 4096 rows without 13.1 -> 9.6 (50 MB).
constexpr int NR_THREADS = 256;
template <typename OT, int CH, bool RES>
__global__ void __launch_bounds__(NR_THREADS) norm_rows4_kernel(float* __restrict__ x, const float* __restrict__ v, long long ldv,
                                                                const float* __restrict__ w, OT* __restrict__ out,
                                                                long long ldo, int n, float eps, float scale) {
  __shared__ float red[33];
  pdl_wait();
  pdl_launch_dependents();
  const float4 *vr = (const float4*)(v + (size_t)blockIdx.x * ldv), *w4 = (const float4*)w;
  float4* row = (float4*)(x + (size_t)blockIdx.x * n);
  OT* dst = out + (size_t)blockIdx.x * ldo;
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 a[CH], b[CH], g[CH];
  float sq = 0.f;
#pragma unroll
  for (int k = 0; k < CH; k++) {
    const int i = threadIdx.x + k * NR_THREADS;
    const bool on = i < n / 4;
    a[k] = on ? vr[i] : z;
    if (RES) b[k] = on ? row[i] : z;
    g[k] = on ? w4[i] : z;
  }
#pragma unroll
  for (int k = 0; k < CH; k++) sq = sq4(a[k], sq);
  sq = block_sum(sq, red);
  const float r = rsqrtf(sq / n + eps) * scale;
#pragma unroll
  for (int k = 0; k < CH; k++) {
    const int i = threadIdx.x + k * NR_THREADS;
    if (i >= n / 4) continue;
    float4 y;
    if (RES) {
      y = make_float4(fmaf(a[k].x * r, g[k].x, b[k].x), fmaf(a[k].y * r, g[k].y, b[k].y), fmaf(a[k].z * r, g[k].z, b[k].z),
                      fmaf(a[k].w * r, g[k].w, b[k].w));
      row[i] = y;
    } else {
      y = make_float4(a[k].x * r * g[k].x, a[k].y * r * g[k].y, a[k].z * r * g[k].z, a[k].w * r * g[k].w);
    }
    st4(dst + i * 4, y);
  }
}
// whole 16-byte pieces and no more of them than a block holds
template <typename OT>
bool norm_rows4_takes(const void* x, const void* v, long long ldv, const void* w, const void* out, long long ldo, int n) {
  return n % 4 == 0 && n <= 4 * 4 * NR_THREADS && ldv % 4 == 0 && ldo % 4 == 0 &&
         (((uintptr_t)x | (uintptr_t)v | (uintptr_t)w) & 15) == 0 && (uintptr_t)out % (4 * sizeof(OT)) == 0;
}
template <typename OT, bool RES>
int norm_rows4_launch(float* x, const float* v, long long ldv, const float* w, OT* out, long long ldo, int n, float eps,
                      float scale, int rows, cudaStream_t s) {
  LaunchCfg lc(dim3(rows), dim3(NR_THREADS), 0, s, pdl_enabled());
  if (n <= 4 * NR_THREADS)
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, norm_rows4_kernel<OT, 1, RES>, x, v, ldv, w, out, ldo, n, eps, scale));
  else if (n <= 8 * NR_THREADS)
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, norm_rows4_kernel<OT, 2, RES>, x, v, ldv, w, out, ldo, n, eps, scale));
  else
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, norm_rows4_kernel<OT, 4, RES>, x, v, ldv, w, out, ldo, n, eps, scale));
  return TLB_OK;
}

// x += norm(y) * w, the sum also as the next product's operand; without y only the latter
constexpr int RR_HOLD = 8;    // values of y a thread keeps between the passes
template <typename OT>
__global__ void __launch_bounds__(512) residual_rows_kernel(float* __restrict__ x, const float* __restrict__ y,
                                                            const float* __restrict__ w, OT* __restrict__ out,
                                                            long long ldo, int n, float eps) {
  __shared__ float red[33];
  pdl_wait();
  pdl_launch_dependents();
  float* row = x + (size_t)blockIdx.x * n;
  OT* dst = out + (size_t)blockIdx.x * ldo;
  if (!y) {
    for (int i = threadIdx.x; i < n; i += 512) put(dst + i, row[i]);
    return;
  }
  const float* yr = y + (size_t)blockIdx.x * n;
  float v[RR_HOLD], sq = 0.f;
#pragma unroll
  for (int k = 0; k < RR_HOLD; k++) {
    const int i = threadIdx.x + k * 512;
    v[k] = i < n ? yr[i] : 0.f;
    sq = fmaf(v[k], v[k], sq);
  }
  for (int i = threadIdx.x + RR_HOLD * 512; i < n; i += 512) sq = fmaf(yr[i], yr[i], sq);
  sq = block_sum(sq, red);
  const float r = rsqrtf(sq / n + eps);
#pragma unroll
  for (int k = 0; k < RR_HOLD; k++) {
    const int i = threadIdx.x + k * 512;
    if (i < n) {
      const float s = fmaf(v[k] * r, w[i], row[i]);
      row[i] = s;
      put(dst + i, s);
    }
  }
  for (int i = threadIdx.x + RR_HOLD * 512; i < n; i += 512) {
    const float s = fmaf(yr[i] * r, w[i], row[i]);
    row[i] = s;
    put(dst + i, s);
  }
}

// 1024 columns a block
template <typename WT>
__global__ void embed_scaled_kernel(const WT* __restrict__ embed, long long ld, const int* __restrict__ ids,
                                    float* __restrict__ x, int width, float scale) {
  pdl_wait();
  pdl_launch_dependents();
  const WT* src = embed + (size_t)ids[blockIdx.x] * ld;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int i = blockIdx.y * 1024 + k * 256 + threadIdx.x;
    if (i < width) x[(size_t)blockIdx.x * width + i] = to_f(src[i]) * scale;
  }
}

__global__ void gather_rows_kernel(const float* __restrict__ x, const int* __restrict__ idx, float* __restrict__ out,
                                   int width) {
  pdl_wait();
  pdl_launch_dependents();
  const float* src = x + (size_t)idx[blockIdx.x] * width;
  for (int i = threadIdx.x; i < width; i += blockDim.x) out[(size_t)blockIdx.x * width + i] = src[i];
}

__global__ void glu_rows_kernel(const float* __restrict__ gu, float* __restrict__ out, long long n, float limit) {
  pdl_wait();
  pdl_launch_dependents();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 v = ((const float2*)gu)[i];
    out[i] = glu_clipped(v.x, v.y, limit);
  }
}

__global__ void relu2_rows_kernel(const float* __restrict__ u, float* __restrict__ out, long long n) {
  pdl_wait();
  pdl_launch_dependents();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = relu2(u[i]);
}

}  // namespace

int row_gemv_launch(DeviceCtx* c, const RowGemv& p, bool bf16, cudaStream_t s) {
  return bf16 ? rg_plan_launch<__nv_bfloat16>(c, p, s) : rg_plan_launch<float>(c, p, s);
}

int rms_rows_launch(const float* x, long long ldx, const float* w, void* out, long long ldo, int n, float eps,
                    float scale, int rows, bool bf16, cudaStream_t s) {
  if (bf16 && norm_rows4_takes<__nv_bfloat16>(nullptr, x, ldx, w, out, ldo, n))
    return norm_rows4_launch<__nv_bfloat16, false>(nullptr, x, ldx, w, (__nv_bfloat16*)out, ldo, n, eps, scale, rows, s);
  if (!bf16 && norm_rows4_takes<float>(nullptr, x, ldx, w, out, ldo, n))
    return norm_rows4_launch<float, false>(nullptr, x, ldx, w, (float*)out, ldo, n, eps, scale, rows, s);
  LaunchCfg lc(dim3(rows), dim3(256), 0, s, pdl_enabled());
  if (bf16)
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, rms_rows_kernel<__nv_bfloat16>, x, ldx, w, (__nv_bfloat16*)out, ldo, n, eps, scale));
  else
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, rms_rows_kernel<float>, x, ldx, w, (float*)out, ldo, n, eps, scale));
  return TLB_OK;
}

int residual_rows_launch(float* x, const float* y, const float* w, void* out, long long ldo, int n, float eps, int rows,
                         bool bf16, cudaStream_t s) {
  if (y && bf16 && norm_rows4_takes<__nv_bfloat16>(x, y, n, w, out, ldo, n))
    return norm_rows4_launch<__nv_bfloat16, true>(x, y, n, w, (__nv_bfloat16*)out, ldo, n, eps, 1.f, rows, s);
  if (y && !bf16 && norm_rows4_takes<float>(x, y, n, w, out, ldo, n))
    return norm_rows4_launch<float, true>(x, y, n, w, (float*)out, ldo, n, eps, 1.f, rows, s);
  LaunchCfg lc(dim3(rows), dim3(512), 0, s, pdl_enabled());
  if (bf16)
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, residual_rows_kernel<__nv_bfloat16>, x, y, w, (__nv_bfloat16*)out, ldo, n, eps));
  else
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, residual_rows_kernel<float>, x, y, w, (float*)out, ldo, n, eps));
  return TLB_OK;
}

int relu2_rows_launch(const float* u, float* out, int ff, int rows, cudaStream_t s) {
  const long long n = (long long)rows * ff, b = (n + 255) / 256;
  LaunchCfg lc(dim3((unsigned)(b < 148 * 16 ? b : 148 * 16)), dim3(256), 0, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, relu2_rows_kernel, u, out, n));
  return TLB_OK;
}

int embed_scaled_launch(const void* embed, const int* ids, float* x, int width, long long ld, float scale, int rows,
                        bool bf16, cudaStream_t s) {
  LaunchCfg lc(dim3(rows, (width + 1023) / 1024), dim3(256), 0, s, pdl_enabled());
  if (bf16) TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, embed_scaled_kernel<__nv_bfloat16>, (const __nv_bfloat16*)embed, ld, ids, x, width, scale));
  else TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, embed_scaled_kernel<float>, (const float*)embed, ld, ids, x, width, scale));
  return TLB_OK;
}

int gather_rows_launch(const float* x, const int* idx, float* out, int width, int rows, cudaStream_t s) {
  LaunchCfg lc(dim3(rows), dim3(256), 0, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, gather_rows_kernel, x, idx, out, width));
  return TLB_OK;
}

int glu_rows_launch(const float* gu, float* out, int ff, float limit, int rows, cudaStream_t s) {
  const long long n = (long long)rows * ff;
  const long long b = (n + 255) / 256;
  LaunchCfg lc(dim3((unsigned)(b < 148 * 16 ? b : 148 * 16)), dim3(256), 0, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, glu_rows_kernel, gu, out, n, limit));
  return TLB_OK;
}

}  // namespace tlb
