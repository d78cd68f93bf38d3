// The recurrences of a prompt pass in chunks of 64 tokens on the tensor pipe (bf16 models; widths that
// are multiples of 8, state width up to 128).  With b_t the running sum of log decays inside a chunk and
// S the state in front of it, both recurrences are
//   O_t = exp(b_t) q_t S + sum_{s <= t} exp(b_t - b_s) (q_t . k_s) u_s
//   S  <- exp(b_L) S + sum_s exp(b_L - b_s) k_s u_s^T
// with u_s = dt_s x_s for ssd, and for the delta rule U = T (V - exp(b) (K S)), where
// T = (I + A)^-1 diag(beta), A_ts = beta_t exp(b_t - b_s) (k_t . k_s) below the diagonal
// (the chunk-parallel form of DeltaNet, Yang et al., "Parallelizing Linear Transformers with the Delta
// Rule over Sequence Length").
//
// What the short convolutions leave (q, k, v) is bf16 and enters the products exactly; everything else
// -- unit norms, step sizes, decays, T, U, the state -- is f32: as factors of rows and columns outside
// the products, or as operands split into two bf16 planes (hi + lo).  The state stays in f32
// accumulators for the whole pass.
//
//   delta_solve   (chunk, head): T of every chunk, in two planes
//   delta_chunk   (32 or 16 value columns, head): the chunks in order
//   ssd_chunk     (32 value columns, head, segment): a segment's chunks in order
//   ssd_state     the same grid: what a segment adds to the state, without its outputs
//
// The delta rule is one segment.  The state of ssd only decays by a scalar between two places, so a long prompt
// is cut into segments that run at once: ssd_state first leaves each segment's own state and log decay, and
// ssd_chunk starts from what the segments in front add up to.  One walk over the chunks has four warps an SM
// and waits on its own latencies; three CTAs an SM and the second, shorter walk take less: 4096 tokens, 64 heads of
// 128 x 64, 44 + 138 us in three segments (53 + 174 with divisions in the copies and branches around the exponentials; two
// CTAs an SM, every buffer doubled, 53 + 228 in eight; 320 in one walk).
#include "mixers.cuh"
#include "rows_mma.cuh"

namespace tlb {

namespace {

constexpr int RC_MOST = 8;   // segments
// CTAs of both ssd kernels that an SM holds, and the most of them an SM that segments may come to: under three rounds
constexpr int RC_PLACES = 3, RC_CTAS_MOST = 8;
constexpr int RC_L = 64, RC_E = 32, RC_THREADS = 128;
constexpr int RC_TLD = RC_L + 8, RC_ELD = RC_E + 8;

// b_t of the chunk (lanes hold tokens lane and lane + 32) from the rates x_t = -log g_t
__device__ __forceinline__ void rc_scan(float x0, float x1, float& b0, float& b1) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y0 = __shfl_up_sync(0xffffffffu, x0, o), y1 = __shfl_up_sync(0xffffffffu, x1, o);
    if (lane >= o) { x0 += y0; x1 += y1; }
  }
  x1 += __shfl_sync(0xffffffffu, x0, 31);
  b0 = -x0;
  b1 = -x1;
}

// Rows t0 .. of a chunk (n of its 64, zeros behind them): `chunks` of the CPR 16-byte pieces of a row of shared memory, by
// RC_THREADS threads.  A thread keeps its piece: no division (those of runtime widths were a third of a chunk's time).
template <int CPR>
__device__ __forceinline__ void rc_fetch(__nv_bfloat16* dst, int ld, const __nv_bfloat16* src, long long row, int chunks, int n, int tid) {
  const int c = tid % CPR;
  if (c >= chunks) return;
#pragma unroll
  for (int i = 0; i < RC_L * CPR / RC_THREADS; i++) {
    const int r = tid / CPR + i * (RC_THREADS / CPR);
    rc_cp16(dst + r * ld + c * 8, src + (r < n ? r : 0) * row + c * 8, r < n);
  }
}
// x exp(d) f where `on`, else zero, without a branch around the exponential (a hundred cycles an element with one)
__device__ __forceinline__ float rc_decayed(float x, float d, float f, bool on) {
  const float y = x * (expf(on ? d : 0.f) * f);
  return on ? y : 0.f;
}

// ---- T of one chunk and head -----------------------------------------------------------------
template <int DP>
__global__ void __launch_bounds__(RC_THREADS) delta_solve_kernel(const __grid_constant__ RecurP p,
                                                                 const __nv_bfloat16* __restrict__ conv,
                                                                 const float2* __restrict__ gates,
                                                                 const float2* __restrict__ norms,
                                                                 __nv_bfloat16* __restrict__ T, int rows) {
  constexpr int LD = DP + 8, AL = RC_L + 1;
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* ks = (__nv_bfloat16*)smem;              // [64][LD]
  float* A = (float*)(smem + (size_t)RC_L * LD * 2);     // [64][AL]
  float* X = A + RC_L * AL;                              // [64][AL]
  float* P = X + RC_L * AL;                              // [3][16][17]
  __shared__ float sb[RC_L], sbeta[RC_L], sn[RC_L];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t0 = blockIdx.x * RC_L, h = blockIdx.y, kg = h / (p.H / p.G), n = rows - t0 < RC_L ? rows - t0 : RC_L;
  for (int i = tid; i < RC_L * LD / 8; i += RC_THREADS) ((uint4*)ks)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < RC_L * AL; i += RC_THREADS) X[i] = 0.f;
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  rc_fetch<DP / 8>(ks, LD, conv + (size_t)t0 * p.cv.C + p.ck + kg * p.D, p.cv.C, p.D / 8, n, tid);
  rc_commit();
  if (warp == 0) {
    const float2 z = make_float2(0.f, 0.f);
    const float2 g0 = lane < n ? gates[(size_t)(t0 + lane) * p.H + h] : z;
    const float2 g1 = lane + 32 < n ? gates[(size_t)(t0 + lane + 32) * p.H + h] : z;
    float b0, b1;
    rc_scan(g0.y, g1.y, b0, b1);
    sb[lane] = b0; sb[lane + 32] = b1;
    sbeta[lane] = g0.x; sbeta[lane + 32] = g1.x;
    sn[lane] = lane < n ? norms[(size_t)(t0 + lane) * p.G + kg].y : 0.f;
    sn[lane + 32] = lane + 32 < n ? norms[(size_t)(t0 + lane + 32) * p.G + kg].y : 0.f;
  }
  rc_wait<0>();
  __syncthreads();
  float s[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
  for (int k = 0; k < DP; k += 16) {
    uint32_t a[4], b[4];
    rc_ldm(a, rc_a(ks, LD, warp * 16, k, lane));
#pragma unroll
    for (int j = 0; j < 4; j++) {
      rc_ldm(b, rc_bn(ks, LD, j * 16, k, lane));
      rc_mma(s[2 * j], a, b[0], b[1]);
      rc_mma(s[2 * j + 1], a, b[2], b[3]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int t = warp * 16 + (lane >> 2) + (e >> 1) * 8, c = j * 8 + (lane & 3) * 2 + (e & 1);
      A[t * AL + c] = c < t ? s[j][e] * sn[t] * sn[c] * sbeta[t] * expf(sb[t] - sb[c]) : 0.f;
    }
  __syncthreads();
  // (I + A)^-1 in blocks of 16: the diagonal blocks column by column, then the blocks below, one
  // block diagonal after the other: X_ij = -X_ii sum_{j <= k < i} A_ik X_kj
  if (tid < 64) {
    const int o = (tid >> 4) * 16, c = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      float v = i == c ? 1.f : 0.f;
#pragma unroll
      for (int k = 0; k < i; k++) v = fmaf(-A[(o + i) * AL + o + k], x[k], v);
      x[i] = v;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) X[(o + i) * AL + o + c] = x[i];
  }
  for (int d = 1; d < 4; d++) {
    __syncthreads();
    for (int i = tid; i < (4 - d) * 256; i += RC_THREADS) {
      const int blk = i >> 8, r = (i >> 4) & 15, c = i & 15, bi = blk + d, bj = blk;
      float v = 0.f;
      for (int k = bj * 16; k < bi * 16; k++) v = fmaf(A[(bi * 16 + r) * AL + k], X[k * AL + bj * 16 + c], v);
      P[(blk * 16 + r) * 17 + c] = v;
    }
    __syncthreads();
    for (int i = tid; i < (4 - d) * 256; i += RC_THREADS) {
      const int blk = i >> 8, r = (i >> 4) & 15, c = i & 15, bi = blk + d, bj = blk;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < 16; k++) v = fmaf(X[(bi * 16 + r) * AL + bi * 16 + k], P[(blk * 16 + k) * 17 + c], v);
      X[(bi * 16 + r) * AL + bj * 16 + c] = -v;
    }
  }
  __syncthreads();
  __nv_bfloat16* out = T + ((size_t)blockIdx.x * p.H + h) * 2 * RC_L * RC_L;
  for (int i = tid; i < RC_L * RC_L / 2; i += RC_THREADS) {
    const int r = i / (RC_L / 2), c = (i % (RC_L / 2)) * 2;
    uint32_t hi, lo;
    rc_split(X[r * AL + c] * sbeta[c], X[r * AL + c + 1] * sbeta[c + 1], hi, lo);
    ((uint32_t*)out)[i] = hi;
    ((uint32_t*)(out + RC_L * RC_L))[i] = lo;
  }
}

// ---- delta rule: the chunks of one head and CE value columns -----------------------------------------------
// One chunk's state is the next one's input, and what costs is that chain: k S, T R and the state's update, with a barrier
// between each.  Four warps walk it; four others take q S, q k^T and the outputs beside it, and are behind them by what they
// have to do alone: named barriers tell them that U is there, and the walk that the state's planes are read.  4096 tokens,
// 16 heads of 128 x 128: four warps for all of it 326 us, eight 282; without branches around the exponentials and waits for
// the next chunk's scalars 208, without divisions in the copies 200.
constexpr int RD_THREADS = 2 * RC_THREADS;
__device__ __forceinline__ void rd_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }   // the four warps of the state
// U of a chunk is there (2), its state's planes are read (3): four warps arrive and go on, the others wait
template <int ID> __device__ __forceinline__ void rd_arrive() { asm volatile("bar.arrive %0, 256;" ::"n"(ID) : "memory"); }
template <int ID> __device__ __forceinline__ void rd_await() { asm volatile("bar.sync %0, 256;" ::"n"(ID) : "memory"); }
template <int DP, int CE>
struct RcSmem {
  static constexpr int LD = DP + 8;
  static constexpr size_t K = 0;                                            // [2][64][LD]
  static constexpr size_t Q = K + (size_t)2 * RC_L * LD * 2;
  static constexpr size_t X = Q + (size_t)2 * RC_L * LD * 2;                // [2][64][ELD]
  static constexpr size_t S = X + (size_t)2 * RC_L * (CE + 8) * 2;            // [2 planes][DP][ELD]
  static constexpr size_t W = S + (size_t)2 * DP * (CE + 8) * 2;              // [2 planes][64][ELD]
  static constexpr size_t U = W + (size_t)2 * RC_L * (CE + 8) * 2;            // [2 planes][64][ELD]
  static constexpr size_t T = U + (size_t)2 * RC_L * (CE + 8) * 2;            // [2][2 planes][64][TLD]
  static constexpr size_t SC = T + (size_t)4 * RC_L * RC_TLD * 2;             // [2][3][64] f32
  static constexpr size_t TOTAL = SC + 2 * 3 * RC_L * 4;
};

template <int DP, int CE>
__global__ void __launch_bounds__(RD_THREADS, 1)
    delta_chunk_kernel(const __grid_constant__ RecurP p, const __nv_bfloat16* __restrict__ conv,
                       const float2* __restrict__ gates, const float2* __restrict__ norms,
                       const __nv_bfloat16* __restrict__ T, float* __restrict__ o, int rows, int pos0) {
  using SM = RcSmem<DP, CE>;
  constexpr int LD = SM::LD, MT = DP / 64, NT = CE / 8;   // state row tiles of 16 per warp, column tiles
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* ksm = (__nv_bfloat16*)(smem + SM::K);
  __nv_bfloat16* qsm = (__nv_bfloat16*)(smem + SM::Q);
  __nv_bfloat16* xsm = (__nv_bfloat16*)(smem + SM::X);
  __nv_bfloat16* ssm = (__nv_bfloat16*)(smem + SM::S);
  __nv_bfloat16* wsm = (__nv_bfloat16*)(smem + SM::W);
  __nv_bfloat16* usm = (__nv_bfloat16*)(smem + SM::U);
  __nv_bfloat16* tsm = (__nv_bfloat16*)(smem + SM::T);
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 3, wr = warp * 16;   // rows of the chunk and of the state
  const bool outs = tid >= RC_THREADS;
  const int h = blockIdx.y, c0 = blockIdx.x * CE, kg = h / (p.H / p.G), D = p.D, E = p.E;
  const int nch = (rows + RC_L - 1) / RC_L;
  const int dch = D / 8, ech = (E - c0 < CE ? E - c0 : CE) / 8;
  for (int i = tid; i < (int)(SM::SC / 16); i += RD_THREADS) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  // (the warps of the state fetch and scan: the others have more to do)
  auto fetch = [&](int ch, int buf) {
    const int t0 = ch * RC_L, n = rows - t0 < RC_L ? rows - t0 : RC_L;
    const __nv_bfloat16* row = conv + (size_t)t0 * p.cv.C;
    rc_fetch<DP / 8>(ksm + buf * RC_L * LD, LD, row + p.ck + kg * D, p.cv.C, dch, n, tid);
    rc_fetch<DP / 8>(qsm + buf * RC_L * LD, LD, row + p.cq + kg * D, p.cv.C, dch, n, tid);
    rc_fetch<CE / 8>(xsm + buf * RC_L * (CE + 8), CE + 8, row + p.cvv + h * E + c0, p.cv.C, ech, n, tid);
    rc_fetch<RC_L / 8>(tsm + (size_t)buf * 2 * RC_L * RC_TLD, RC_TLD, T + ((size_t)ch * p.H + h) * 2 * RC_L * RC_L, RC_L, RC_L / 8, RC_L, tid);
    rc_fetch<RC_L / 8>(tsm + ((size_t)buf * 2 + 1) * RC_L * RC_TLD, RC_TLD, T + (((size_t)ch * p.H + h) * 2 + 1) * RC_L * RC_L, RC_L, RC_L / 8, RC_L, tid);
  };
  // one of them carries the next chunk's scalars in registers (tokens lane and lane + 32)
  float2 g0, g1, n0, n1;
  // (the last row's for tokens behind it, zeroed where they are used: nothing waits for a load here)
  auto scalars = [&](int ch) {
    const int t0 = ch * RC_L + lane < rows ? ch * RC_L + lane : rows - 1, t1 = ch * RC_L + lane + 32 < rows ? ch * RC_L + lane + 32 : rows - 1;
    g0 = gates[(size_t)t0 * p.H + h];
    g1 = gates[(size_t)t1 * p.H + h];
    n0 = norms[(size_t)t0 * p.G + kg];
    n1 = norms[(size_t)t1 * p.G + kg];
  };
  // state: this warp's rows of it, CE columns, as accumulators
  float s[MT][NT][4];
  float* S = p.S + (size_t)h * D * E;
  auto state_at = [&](int mt, int nt, int e, int& r, int& c) {
    r = (warp * MT + mt) * 16 + (lane >> 2) + (e >> 1) * 8;
    c = c0 + nt * 8 + (lane & 3) * 2 + (e & 1);
  };
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int r, c;
        state_at(mt, nt, e, r, c);
        s[mt][nt][e] = !outs && pos0 > 0 && r < D && c < E ? S[(size_t)r * E + c] : 0.f;
      }
  if (!outs) {
    fetch(0, 0);
    rc_commit();
    if (warp == 0) scalars(0);
  }
  for (int ch = 0; ch < nch; ch++) {
    const int buf = ch & 1, t0 = ch * RC_L, n = rows - t0 < RC_L ? rows - t0 : RC_L;
    float* sb = (float*)(smem + SM::SC) + buf * 3 * RC_L;   // b_t
    float* snk = sb + RC_L;                                 // 1 / |k_s|
    float* snq = snk + RC_L;                                // D^-1/2 / |q_t|
    if (!outs) {
      // the state in front of the chunk, in two planes, for the products below
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            uint32_t hi, lo;
            rc_split(s[mt][nt][2 * e], s[mt][nt][2 * e + 1], hi, lo);
            const int at = ((warp * MT + mt) * 16 + (lane >> 2) + e * 8) * (CE + 8) + nt * 8 + (lane & 3) * 2;
            *(uint32_t*)(ssm + at) = hi;
            *(uint32_t*)(ssm + DP * (CE + 8) + at) = lo;
          }
    }
    if (warp == 0 && !outs) {
      float b0, b1;
      const bool on0 = lane < n, on1 = lane + 32 < n;
      rc_scan(on0 ? g0.y : 0.f, on1 ? g1.y : 0.f, b0, b1);
      sb[lane] = b0; sb[lane + 32] = b1;
      snk[lane] = on0 ? n0.y : 0.f; snk[lane + 32] = on1 ? n1.y : 0.f;
      snq[lane] = on0 ? n0.x : 0.f; snq[lane + 32] = on1 ? n1.x : 0.f;
      if (ch + 1 < nch) scalars(ch + 1);
    }
    rc_wait<0>();
    __syncthreads();   // the chunk's rows and the state's planes are there
    const __nv_bfloat16 *K = ksm + buf * RC_L * LD, *Q = qsm + buf * RC_L * LD, *X = xsm + buf * RC_L * (CE + 8);
    const int ra = wr + (lane >> 2), cb = (lane & 3) * 2;     // the thread's rows are ra and ra + 8
    const float ba = sb[ra], bb = sb[ra + 8], bL = sb[RC_L - 1];
    const float qa = snq[ra], qb = snq[ra + 8];
    if (!outs) {
      if (ch + 1 < nch) {
        fetch(ch + 1, buf ^ 1);
        rc_commit();
      }
      // k S (both planes of S)
      // (a plane or a product of planes has sums of its own: their chains run side by side)
      float kS[2][NT][4];
#pragma unroll
      for (int i = 0; i < NT; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) kS[0][i][e] = kS[1][i][e] = 0.f;
#pragma unroll
      for (int k = 0; k < DP; k += 16) {
        uint32_t ak[4], bs[2][CE / 16][4];
        rc_ldm(ak, rc_a(K, LD, wr, k, lane));
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++) rc_ldmt(bs[pl][j], rc_bk(ssm + pl * DP * (CE + 8), (CE + 8), k, j * 16, lane));
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++) {
            rc_mma(kS[pl][2 * j], ak, bs[pl][j][0], bs[pl][j][1]);
            rc_mma(kS[pl][2 * j + 1], ak, bs[pl][j][2], bs[pl][j][3]);
          }
      }
      // R = v - exp(b) |k|^-1 (k S), in planes
      const float fa = expf(ba) * snk[ra], fb = expf(bb) * snk[ra + 8];
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int at = (ra + 8 * e) * (CE + 8) + j * 8 + cb;
          const uint32_t v = *(const uint32_t*)(X + at);
          const float f = e ? fb : fa;
          uint32_t hi, lo;
          rc_split(fmaf(-f, kS[0][j][2 * e] + kS[1][j][2 * e], __uint_as_float(v << 16)),
                   fmaf(-f, kS[0][j][2 * e + 1] + kS[1][j][2 * e + 1], __uint_as_float(v & 0xffff0000u)), hi, lo);
          *(uint32_t*)(usm + at) = hi;
          *(uint32_t*)(usm + RC_L * (CE + 8) + at) = lo;
        }
      rd_sync();
      float u[NT][4], uc[2][NT][4];
#pragma unroll
      for (int i = 0; i < NT; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) u[i][e] = uc[0][i][e] = uc[1][i][e] = 0.f;
      const __nv_bfloat16* Tp = tsm + (size_t)buf * 2 * RC_L * RC_TLD;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k <= warp) {
          uint32_t ah[4], al[4];
          rc_ldm(ah, rc_a(Tp, RC_TLD, wr, k * 16, lane));
          rc_ldm(al, rc_a(Tp + RC_L * RC_TLD, RC_TLD, wr, k * 16, lane));
#pragma unroll
          for (int j = 0; j < CE / 16; j++) {
            uint32_t bh[4], bl[4];
            rc_ldmt(bh, rc_bk(usm, (CE + 8), k * 16, j * 16, lane));
            rc_ldmt(bl, rc_bk(usm + RC_L * (CE + 8), (CE + 8), k * 16, j * 16, lane));
            rc_mma(u[2 * j], ah, bh[0], bh[1]); rc_mma(u[2 * j + 1], ah, bh[2], bh[3]);
            rc_mma(uc[0][2 * j], ah, bl[0], bl[1]); rc_mma(uc[0][2 * j + 1], ah, bl[2], bl[3]);
            rc_mma(uc[1][2 * j], al, bh[0], bh[1]); rc_mma(uc[1][2 * j + 1], al, bh[2], bh[3]);
          }
        }
#pragma unroll
      for (int i = 0; i < NT; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) u[i][e] += uc[0][i][e] + uc[1][i][e];
      rd_sync();   // R is read: its planes become U's
      const float ga = expf(bL - ba) * snk[ra], gb = expf(bL - bb) * snk[ra + 8];
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int at = (ra + 8 * e) * (CE + 8) + j * 8 + cb;
          const float f = e ? gb : ga;
          uint32_t hi, lo;
          rc_split(u[j][2 * e], u[j][2 * e + 1], hi, lo);
          *(uint32_t*)(usm + at) = hi;
          *(uint32_t*)(usm + RC_L * (CE + 8) + at) = lo;
          rc_split(u[j][2 * e] * f, u[j][2 * e + 1] * f, hi, lo);
          *(uint32_t*)(wsm + at) = hi;
          *(uint32_t*)(wsm + RC_L * (CE + 8) + at) = lo;
        }
      rd_arrive<2>();
      rd_sync();   // the weighted form is there
      // S = exp(b_L) S + K^T (weighted U)
      const float eL = expf(bL);
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) s[mt][nt][e] *= eL;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        uint32_t a[MT][4];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) rc_ldmt(a[mt], rc_at(K, LD, (warp * MT + mt) * 16, k * 16, lane));
        uint32_t b[2][CE / 16][4];
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++) rc_ldmt(b[pl][j], rc_bk(wsm + pl * RC_L * (CE + 8), (CE + 8), k * 16, j * 16, lane));
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++)
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
              rc_mma(s[mt][2 * j], a[mt], b[pl][j][0], b[pl][j][1]);
              rc_mma(s[mt][2 * j + 1], a[mt], b[pl][j][2], b[pl][j][3]);
            }
      }
      rd_await<3>();   // before the next chunk's planes
    } else {
      float qs[NT][4];
      uint32_t mh[4][4], ml[4][4];
      // q S (both planes of S)
#pragma unroll
      for (int i = 0; i < NT; i++) qs[i][0] = qs[i][1] = qs[i][2] = qs[i][3] = 0.f;
#pragma unroll
      for (int k = 0; k < DP; k += 16) {
        uint32_t aq[4], bs[2][CE / 16][4];
        rc_ldm(aq, rc_a(Q, LD, wr, k, lane));
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++) rc_ldmt(bs[pl][j], rc_bk(ssm + pl * DP * (CE + 8), (CE + 8), k, j * 16, lane));
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
          for (int j = 0; j < CE / 16; j++) {
            rc_mma(qs[2 * j], aq, bs[pl][j][0], bs[pl][j][1]);
            rc_mma(qs[2 * j + 1], aq, bs[pl][j][2], bs[pl][j][3]);
          }
      }
      rd_arrive<3>();
      // q k^T
      float m[8][4];
#pragma unroll
      for (int i = 0; i < 8; i++) m[i][0] = m[i][1] = m[i][2] = m[i][3] = 0.f;
#pragma unroll
      for (int k = 0; k < DP; k += 16) {
        uint32_t aq[4], bk[4][4];   // all of a step's fragments first: one shared-memory latency a step
        rc_ldm(aq, rc_a(Q, LD, wr, k, lane));
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (j <= warp) rc_ldm(bk[j], rc_bn(K, LD, j * 16, k, lane));
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (j <= warp) {
            rc_mma(m[2 * j], aq, bk[j][0], bk[j][1]);
            rc_mma(m[2 * j + 1], aq, bk[j][2], bk[j][3]);
          }
      }
      // decays and unit norms of q k^T, then as operand planes
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j <= 2 * warp + 1) {
          const float2 bc = *(const float2*)(sb + j * 8 + cb), kc = *(const float2*)(snk + j * 8 + cb);
          float w[4];
#pragma unroll
          for (int e = 0; e < 4; e++)
            w[e] = rc_decayed(m[j][e], (e < 2 ? ba : bb) - (e & 1 ? bc.y : bc.x), (e & 1 ? kc.y : kc.x) * (e < 2 ? qa : qb),
                              j * 8 + cb + (e & 1) <= (e < 2 ? ra : ra + 8));
          rc_split(w[0], w[1], mh[j >> 1][(j & 1) * 2], ml[j >> 1][(j & 1) * 2]);
          rc_split(w[2], w[3], mh[j >> 1][(j & 1) * 2 + 1], ml[j >> 1][(j & 1) * 2 + 1]);
        }
      rd_await<2>();
      // O = exp(b) (q S) + M U
      const float ea = expf(ba) * qa, eb = expf(bb) * qb;
#pragma unroll
      for (int j = 0; j < NT; j++) { qs[j][0] *= ea; qs[j][1] *= ea; qs[j][2] *= eb; qs[j][3] *= eb; }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k <= warp) {
#pragma unroll
          for (int j = 0; j < CE / 16; j++) {
            uint32_t b[4];
            rc_ldmt(b, rc_bk(usm, (CE + 8), k * 16, j * 16, lane));
            rc_mma(qs[2 * j], mh[k], b[0], b[1]); rc_mma(qs[2 * j + 1], mh[k], b[2], b[3]);
            rc_mma(qs[2 * j], ml[k], b[0], b[1]); rc_mma(qs[2 * j + 1], ml[k], b[2], b[3]);
            rc_ldmt(b, rc_bk(usm + RC_L * (CE + 8), (CE + 8), k * 16, j * 16, lane));
            rc_mma(qs[2 * j], mh[k], b[0], b[1]); rc_mma(qs[2 * j + 1], mh[k], b[2], b[3]);
          }
        }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int t = ra + 8 * e;
        if (t < n) {
          float* dst = o + ((size_t)(t0 + t) * p.H + h) * E + c0;
#pragma unroll
          for (int j = 0; j < NT; j++)
            if (j < ech) *(float2*)(dst + j * 8 + cb) = make_float2(qs[j][2 * e], qs[j][2 * e + 1]);
        }
      }
    }
  }
  if (outs) return;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int r, c;
        state_at(mt, nt, e, r, c);
        if (r < D && c < E) S[(size_t)r * E + c] = s[mt][nt][e];
      }
}

// Segments of `chunks` chunks each.  carry [segments][H][D][E]: the state in front of the prompt, then every
// segment's own but the last; decay [segments][H]: its log decay.  One segment: no carry.
struct RcSegments {
  int n, chunks;
  float *carry, *decay;
};

// ---- ssd: the chunks of one head and 32 value columns ------------------------------------------------
// The walk waits on its own latencies (mma.sync fragments, barriers, exponentials), so what counts is CTAs an SM: three,
// with every operand once in shared memory.  The next chunk's rows come as their places fall free: q behind q k^T, k
// behind the state's update, which is done before the outputs for that, x behind the next chunk's first barrier.
template <int DP>
struct ScSmem {
  static constexpr int LD = DP + 8;
  static constexpr size_t K = 0;                                            // [64][LD]
  static constexpr size_t Q = K + (size_t)RC_L * LD * 2;
  static constexpr size_t X = Q + (size_t)RC_L * LD * 2;                    // [64][ELD]
  static constexpr size_t S = X + (size_t)RC_L * RC_ELD * 2;                // [2 planes][DP][ELD]
  static constexpr size_t W = S + (size_t)2 * DP * RC_ELD * 2;              // [2 planes][64][ELD]
  static constexpr size_t SC = W + (size_t)2 * RC_L * RC_ELD * 2;           // [2][64] f32
  static constexpr size_t TOTAL = SC + 2 * RC_L * 4;
};

template <int DP>
__global__ void __launch_bounds__(RC_THREADS, RC_PLACES)
    ssd_chunk_kernel(const __grid_constant__ RecurP p, const __nv_bfloat16* __restrict__ conv,
                     const float2* __restrict__ gates, float* __restrict__ o, int rows, int pos0,
                     const __grid_constant__ RcSegments g) {
  using SM = ScSmem<DP>;
  constexpr int LD = SM::LD, MT = DP / 64, NT = RC_E / 8;   // state row tiles of 16 per warp, column tiles
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* K = (__nv_bfloat16*)(smem + SM::K);
  __nv_bfloat16* Q = (__nv_bfloat16*)(smem + SM::Q);
  __nv_bfloat16* X = (__nv_bfloat16*)(smem + SM::X);
  __nv_bfloat16* ssm = (__nv_bfloat16*)(smem + SM::S);
  __nv_bfloat16* wsm = (__nv_bfloat16*)(smem + SM::W);
  float* sb = (float*)(smem + SM::SC);          // b_t
  float* sg = sb + RC_L;                        // dt_s
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wr = warp * 16;
  const int h = blockIdx.y, c0 = blockIdx.x * RC_E, kg = h / (p.H / p.G), D = p.D, E = p.E;
  const int nch = (rows + RC_L - 1) / RC_L, ch0 = (int)blockIdx.z * g.chunks, ch1 = ch0 + g.chunks < nch ? ch0 + g.chunks : nch;
  const int dch = D / 8, ech = (E - c0 < RC_E ? E - c0 : RC_E) / 8;
  for (int i = tid; i < (int)(SM::SC / 16); i += RC_THREADS) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  // rows of a chunk: of k or q from column `at` on, of x
  auto rows_of = [&](int ch) { return rows - ch * RC_L < RC_L ? rows - ch * RC_L : RC_L; };
  auto fetch = [&](__nv_bfloat16* dst, int at, int ch) {
    rc_fetch<DP / 8>(dst, LD, conv + (size_t)ch * RC_L * p.cv.C + at, p.cv.C, dch, rows_of(ch), tid);
    rc_commit();
  };
  auto fetch_x = [&](int ch) {
    rc_fetch<RC_E / 8>(X, RC_ELD, conv + (size_t)ch * RC_L * p.cv.C + p.cvv + h * E + c0, p.cv.C, ech, rows_of(ch), tid);
    rc_commit();
  };
  // warp 0 carries the next chunk's scalars in registers (tokens lane and lane + 32)
  float2 g0, g1;
  // (the last row's for tokens behind it, zeroed where they are used: nothing waits for a load here)
  auto scalars = [&](int ch) {
    const int t0 = ch * RC_L + lane < rows ? ch * RC_L + lane : rows - 1, t1 = ch * RC_L + lane + 32 < rows ? ch * RC_L + lane + 32 : rows - 1;
    g0 = gates[(size_t)t0 * p.H + h];
    g1 = gates[(size_t)t1 * p.H + h];
  };
  fetch(Q, p.cq + kg * D, ch0);
  fetch(K, p.ck + kg * D, ch0);
  if (warp == 0) scalars(ch0);
  // state: this warp's rows of it, 32 columns, as accumulators
  float s[MT][NT][4];
  float* S = p.S + (size_t)h * D * E;
  auto state_at = [&](int mt, int nt, int e, int& r, int& c) {
    r = (warp * MT + mt) * 16 + (lane >> 2) + (e >> 1) * 8;
    c = c0 + nt * 8 + (lane & 3) * 2 + (e & 1);
  };
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int r, c;
        state_at(mt, nt, e, r, c);
        s[mt][nt][e] = pos0 > 0 && g.n == 1 && r < D && c < E ? S[(size_t)r * E + c] : 0.f;
      }
  if (g.n > 1) {
    const size_t HS = (size_t)p.H * D * E;
    for (int j = pos0 > 0 ? 0 : 1; j <= (int)blockIdx.z; j++) {
      const float* C = g.carry + j * HS + (size_t)h * D * E;
      const float f = j > 0 ? expf(g.decay[(j - 1) * p.H + h]) : 0.f;
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            int r, c;
            state_at(mt, nt, e, r, c);
            if (r >= D || c >= E) continue;   // E is even
            const float2 v = __ldcg((const float2*)(C + (size_t)r * E + c));
            s[mt][nt][e] = fmaf(f, s[mt][nt][e], v.x);
            s[mt][nt][e + 1] = fmaf(f, s[mt][nt][e + 1], v.y);
          }
    }
  }
  for (int ch = ch0; ch < ch1; ch++) {
    const int t0 = ch * RC_L, n = rows - t0 < RC_L ? rows - t0 : RC_L;
    // the state in front of the chunk, in two planes, for the products below
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          uint32_t hi, lo;
          rc_split(s[mt][nt][2 * e], s[mt][nt][2 * e + 1], hi, lo);
          const int at = ((warp * MT + mt) * 16 + (lane >> 2) + e * 8) * RC_ELD + nt * 8 + (lane & 3) * 2;
          *(uint32_t*)(ssm + at) = hi;
          *(uint32_t*)(ssm + DP * RC_ELD + at) = lo;
        }
    if (warp == 0) {
      float b0, b1;
      const bool on0 = lane < n, on1 = lane + 32 < n;
      rc_scan(on0 ? g0.y : 0.f, on1 ? g1.y : 0.f, b0, b1);
      sb[lane] = b0; sb[lane + 32] = b1;
      sg[lane] = on0 ? g0.x : 0.f; sg[lane + 32] = on1 ? g1.x : 0.f;
      if (ch + 1 < ch1) scalars(ch + 1);
    }
    rc_wait<0>();
    __syncthreads();   // q, k and the state's planes are there; x of the chunk before is read
    fetch_x(ch);
    const int ra = wr + (lane >> 2), cb = (lane & 3) * 2;     // the thread's rows are ra and ra + 8
    const float ba = sb[ra], bb = sb[ra + 8], bL = sb[RC_L - 1];
    const float ga = expf(bL - ba) * sg[ra], gb = expf(bL - bb) * sg[ra + 8];
    // q S (both planes of S), q k^T for the rows of this warp
    float qs[NT][4], m[8][4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
#pragma unroll
      for (int i = 0; i < NT; i++) qs[i][e] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) m[i][e] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < DP; k += 16) {
      uint32_t aq[4], bs[2][2][4], bk[4][4];   // all of a step's fragments first: one shared-memory latency a step
      rc_ldm(aq, rc_a(Q, LD, wr, k, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++) rc_ldmt(bs[pl][j], rc_bk(ssm + pl * DP * RC_ELD, RC_ELD, k, j * 16, lane));
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j <= warp) rc_ldm(bk[j], rc_bn(K, LD, j * 16, k, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
          rc_mma(qs[2 * j], aq, bs[pl][j][0], bs[pl][j][1]);
          rc_mma(qs[2 * j + 1], aq, bs[pl][j][2], bs[pl][j][3]);
        }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j <= warp) {
          rc_mma(m[2 * j], aq, bk[j][0], bk[j][1]);
          rc_mma(m[2 * j + 1], aq, bk[j][2], bk[j][3]);
        }
    }
    // decays and step sizes of q k^T, then as operand planes
    uint32_t mh[4][4], ml[4][4];
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j <= 2 * warp + 1) {
        const float2 bc = *(const float2*)(sb + j * 8 + cb), gc = *(const float2*)(sg + j * 8 + cb);
        float w[4];
#pragma unroll
        for (int e = 0; e < 4; e++)
          w[e] = rc_decayed(m[j][e], (e < 2 ? ba : bb) - (e & 1 ? bc.y : bc.x), e & 1 ? gc.y : gc.x,
                            j * 8 + cb + (e & 1) <= (e < 2 ? ra : ra + 8));
        rc_split(w[0], w[1], mh[j >> 1][(j & 1) * 2], ml[j >> 1][(j & 1) * 2]);
        rc_split(w[2], w[3], mh[j >> 1][(j & 1) * 2 + 1], ml[j >> 1][(j & 1) * 2 + 1]);
      }
    rc_wait<0>();
    __syncthreads();   // x is there, q is read
    if (ch + 1 < ch1) fetch(Q, p.cq + kg * D, ch + 1);
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int at = (ra + 8 * e) * RC_ELD + j * 8 + cb;
        const uint32_t v = *(const uint32_t*)(X + at);
        const float f = e ? gb : ga;
        uint32_t hi, lo;
        rc_split(f * __uint_as_float(v << 16), f * __uint_as_float(v & 0xffff0000u), hi, lo);
        *(uint32_t*)(wsm + at) = hi;
        *(uint32_t*)(wsm + RC_L * RC_ELD + at) = lo;
      }
    __syncthreads();
    // S = exp(b_L) S + K^T (weighted x)
    const float eL = expf(bL);
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) s[mt][nt][e] *= eL;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t a[MT][4], b[2][2][4];
#pragma unroll
      for (int mt = 0; mt < MT; mt++) rc_ldmt(a[mt], rc_at(K, LD, (warp * MT + mt) * 16, k * 16, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++) rc_ldmt(b[pl][j], rc_bk(wsm + pl * RC_L * RC_ELD, RC_ELD, k * 16, j * 16, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int mt = 0; mt < MT; mt++) {
            rc_mma(s[mt][2 * j], a[mt], b[pl][j][0], b[pl][j][1]);
            rc_mma(s[mt][2 * j + 1], a[mt], b[pl][j][2], b[pl][j][3]);
          }
    }
    __syncthreads();   // k and the weighted x are read
    if (ch + 1 < ch1) fetch(K, p.ck + kg * D, ch + 1);
    // O = exp(b) (q S) + M x
    const float ea = expf(ba), eb = expf(bb);
#pragma unroll
    for (int j = 0; j < NT; j++) { qs[j][0] *= ea; qs[j][1] *= ea; qs[j][2] *= eb; qs[j][3] *= eb; }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k <= warp) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          uint32_t b[4];
          rc_ldmt(b, rc_bk(X, RC_ELD, k * 16, j * 16, lane));
          rc_mma(qs[2 * j], mh[k], b[0], b[1]); rc_mma(qs[2 * j + 1], mh[k], b[2], b[3]);
          rc_mma(qs[2 * j], ml[k], b[0], b[1]); rc_mma(qs[2 * j + 1], ml[k], b[2], b[3]);
        }
      }
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int t = ra + 8 * e;
      if (t < n) {
        float* dst = o + ((size_t)(t0 + t) * p.H + h) * E + c0;
#pragma unroll
        for (int j = 0; j < NT; j++)
          if (j < ech) *(float2*)(dst + j * 8 + cb) = make_float2(qs[j][2 * e], qs[j][2 * e + 1]);
      }
    }
  }
  if ((int)blockIdx.z != g.n - 1) return;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int r, c;
        state_at(mt, nt, e, r, c);
        if (r < D && c < E) S[(size_t)r * E + c] = s[mt][nt][e];
      }
}

// ---- what a segment adds to the state of ssd -------------------------------------------------------
template <int DP>
struct SsSmem {
  static constexpr int LD = DP + 8;
  static constexpr size_t K = 0;                                            // [2][64][LD]
  static constexpr size_t X = K + (size_t)2 * RC_L * LD * 2;                // [2][64][ELD]
  static constexpr size_t W = X + (size_t)2 * RC_L * RC_ELD * 2;            // [2 planes][64][ELD]
  static constexpr size_t SC = W + (size_t)2 * RC_L * RC_ELD * 2;           // [2][64] f32
  static constexpr size_t TOTAL = SC + 2 * RC_L * 4;
};

template <int DP>
__global__ void __launch_bounds__(RC_THREADS, RC_PLACES)
    ssd_state_kernel(const __grid_constant__ RecurP p, const __nv_bfloat16* __restrict__ conv,
                     const float2* __restrict__ gates, int pos0, const __grid_constant__ RcSegments g) {
  using SM = SsSmem<DP>;
  constexpr int LD = SM::LD, MT = DP / 64;
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* ksm = (__nv_bfloat16*)(smem + SM::K);
  __nv_bfloat16* xsm = (__nv_bfloat16*)(smem + SM::X);
  __nv_bfloat16* wsm = (__nv_bfloat16*)(smem + SM::W);
  float* sb = (float*)(smem + SM::SC);
  float* sg = sb + RC_L;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, c0 = blockIdx.x * RC_E, kg = h / (p.H / p.G), D = p.D, E = p.E;
  const int ch0 = (int)blockIdx.z * g.chunks, ch1 = ch0 + g.chunks;   // never the last segment: all chunks whole
  const int dch = D / 8, ech = (E - c0 < RC_E ? E - c0 : RC_E) / 8;
  for (int i = tid; i < (int)(SM::SC / 16); i += RC_THREADS) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  auto fetch = [&](int ch, int buf) {
    const __nv_bfloat16* base = conv + (size_t)ch * RC_L * p.cv.C;
    rc_fetch<DP / 8>(ksm + buf * RC_L * LD, LD, base + p.ck + kg * D, p.cv.C, dch, RC_L, tid);
    rc_fetch<RC_E / 8>(xsm + buf * RC_L * RC_ELD, RC_ELD, base + p.cvv + h * E + c0, p.cv.C, ech, RC_L, tid);
  };
  float2 g0, g1;
  auto scalars = [&](int ch) {
    g0 = gates[(size_t)(ch * RC_L + lane) * p.H + h];
    g1 = gates[(size_t)(ch * RC_L + lane + 32) * p.H + h];
  };
  float s[MT][4][4], total = 0.f;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++) s[mt][nt][0] = s[mt][nt][1] = s[mt][nt][2] = s[mt][nt][3] = 0.f;
  fetch(ch0, 0);
  rc_commit();
  if (warp == 0) scalars(ch0);
  for (int ch = ch0; ch < ch1; ch++) {
    const int buf = (ch - ch0) & 1;
    if (warp == 0) {
      float b0, b1;
      rc_scan(g0.y, g1.y, b0, b1);
      sb[lane] = b0; sb[lane + 32] = b1;
      sg[lane] = g0.x; sg[lane + 32] = g1.x;
      if (ch + 1 < ch1) scalars(ch + 1);
    }
    rc_wait<0>();
    __syncthreads();
    if (ch + 1 < ch1) {
      fetch(ch + 1, buf ^ 1);
      rc_commit();
    }
    const __nv_bfloat16 *K = ksm + buf * RC_L * LD, *X = xsm + buf * RC_L * RC_ELD;
    const float bL = sb[RC_L - 1];
    total += bL;
    // a thread's token, half of its 32 columns: exp(b_L - b_s) dt_s x_s in two planes
    {
      const int t = tid >> 1, at = t * RC_ELD + (tid & 1) * 16;
      const float f = expf(bL - sb[t]) * sg[t];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t v = *(const uint32_t*)(X + at + 2 * i);
        uint32_t hi, lo;
        rc_split(f * __uint_as_float(v << 16), f * __uint_as_float(v & 0xffff0000u), hi, lo);
        *(uint32_t*)(wsm + at + 2 * i) = hi;
        *(uint32_t*)(wsm + RC_L * RC_ELD + at + 2 * i) = lo;
      }
    }
    const float eL = expf(bL);
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int nt = 0; nt < 4; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) s[mt][nt][e] *= eL;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t a[MT][4], b[2][2][4];
#pragma unroll
      for (int mt = 0; mt < MT; mt++) rc_ldmt(a[mt], rc_at(K, LD, (warp * MT + mt) * 16, k * 16, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++) rc_ldmt(b[pl][j], rc_bk(wsm + pl * RC_L * RC_ELD, RC_ELD, k * 16, j * 16, lane));
#pragma unroll
      for (int pl = 0; pl < 2; pl++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int mt = 0; mt < MT; mt++) {
            rc_mma(s[mt][2 * j], a[mt], b[pl][j][0], b[pl][j][1]);
            rc_mma(s[mt][2 * j + 1], a[mt], b[pl][j][2], b[pl][j][3]);
          }
    }
    __syncthreads();   // the chunk's operands and scalars are read: the next one may overwrite them
  }
  const size_t HS = (size_t)p.H * D * E;
  const float* S = p.S + (size_t)h * D * E;
  float* out = g.carry + (blockIdx.z + 1) * HS + (size_t)h * D * E;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int r = (warp * MT + mt) * 16 + (lane >> 2) + (e >> 1) * 8, c = c0 + nt * 8 + (lane & 3) * 2;
        if (r >= D || c >= E) continue;
        *(float2*)(out + (size_t)r * E + c) = make_float2(s[mt][nt][e], s[mt][nt][e + 1]);
        // the next kernel's last segment overwrites the state, so that its others read a copy
        if (blockIdx.z == 0 && pos0 > 0)
          *(float2*)(g.carry + (size_t)h * D * E + (size_t)r * E + c) = *(const float2*)(S + (size_t)r * E + c);
      }
  if (blockIdx.x == 0 && tid == 0) g.decay[blockIdx.z * p.H + h] = total;
}

// Most segments of a prompt (more rows, no fewer): of four chunks at least, since a segment's start reads the states in
// front of it, RC_MOST, and RC_CTAS_MOST CTAs an SM.
int rc_most_segments(const RecurP& p, int rows, int sms) {
  const int nch = (rows + RC_L - 1) / RC_L, ctas = (p.E + RC_E - 1) / RC_E * p.H;
  int n = nch / 4 < RC_MOST ? nch / 4 : RC_MOST;
  if (n * ctas > RC_CTAS_MOST * sms) n = RC_CTAS_MOST * sms / ctas;
  return n < 2 ? 1 : n;
}
// Up to that many, by what they cost: both kernels run in waves of RC_PLACES CTAs an SM, a wave as long as a segment's
// chunks and a start of 1.5 chunks; a chunk of ssd_state takes 0.3 of one of ssd_chunk.  4096 tokens, 64 heads of 128 x 64,
// the 8-layer prompt pass with six such layers, us, the number set by hand: 2 segments 6931, 3 (the rule's) 6470, 4 6816,
// 6 6536, 8 6610, and beyond RC_MOST, which such a number does not repay in scratch, 10 6527, 13 6674, 16 6884.
RcSegments rc_segments(const RecurP& p, int rows, int sms, void* scratch) {
  const int nch = (rows + RC_L - 1) / RC_L, most = rc_most_segments(p, rows, sms), ctas = (p.E + RC_E - 1) / RC_E * p.H;
  RcSegments g{1, nch, nullptr, nullptr};
  long long best = 0;
  for (int want = 1; want <= most; want++) {
    const int chunks = (nch + want - 1) / want, n = (nch + chunks - 1) / chunks;
    auto waves = [&](int segments) { return ((long long)segments * ctas + RC_PLACES * sms - 1) / (RC_PLACES * sms); };
    const long long cost = (10 * waves(n) + 3 * waves(n - 1)) * (2 * chunks + 3);
    if (want > 1 && cost >= best) continue;
    best = cost;
    g.n = n;
    g.chunks = chunks;
  }
  if (g.n == 1) return g;
  g.carry = (float*)scratch;
  g.decay = g.carry + (size_t)g.n * p.H * p.D * p.E;
  return g;
}

template <int DP, int CE>
int delta_walk(const RecurP& p, const void* conv, const float2* gates, const float2* norms, const void* T, float* o, int rows,
               int pos0, cudaStream_t s) {
  constexpr int smem = (int)RcSmem<DP, CE>::TOTAL;
  static std::atomic<unsigned long long> done{0};
  const int rc = ensure_dynamic_smem(delta_chunk_kernel<DP, CE>, smem, done);
  if (rc) return rc;
  LaunchCfg lc(dim3((p.E + CE - 1) / CE, p.H), dim3(RD_THREADS), smem, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, delta_chunk_kernel<DP, CE>, p, (const __nv_bfloat16*)conv, gates, norms,
                              (const __nv_bfloat16*)T, o, rows, pos0));
  return TLB_OK;
}

template <int DP>
int delta_launch(const RecurP& p, const void* conv, const float2* gates, const float2* norms, void* T, float* o, int rows,
                 int pos0, cudaStream_t s) {
  DeviceCtx* c = nullptr;
  int rc = get_ctx(&c);
  if (rc) return rc;
  constexpr int smem = RC_L * (DP + 8) * 2 + (2 * RC_L * (RC_L + 1) + 3 * 16 * 17) * 4;
  static std::atomic<unsigned long long> done{0};
  rc = ensure_dynamic_smem(delta_solve_kernel<DP>, smem, done);
  if (rc) return rc;
  LaunchCfg lc(dim3((rows + RC_L - 1) / RC_L, p.H), dim3(RC_THREADS), smem, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, delta_solve_kernel<DP>, p, (const __nv_bfloat16*)conv, gates, norms,
                              (__nv_bfloat16*)T, rows));
  // few heads: half as many columns a CTA, twice the CTAs, where those still find an SM each (4096 tokens, 16 heads of
  // 128, before the outputs had warps of their own: 392 us on 64 SMs, 318 on 128)
  if (2 * ((p.E + RC_E - 1) / RC_E * p.H) <= c->sm_count)
    return delta_walk<DP, 16>(p, conv, gates, norms, T, o, rows, pos0, s);
  return delta_walk<DP, RC_E>(p, conv, gates, norms, T, o, rows, pos0, s);
}

template <int DP>
int ssd_launch(const RecurP& p, const void* conv, const float2* gates, void* scratch, float* o, int rows, int pos0,
               cudaStream_t s) {
  DeviceCtx* c = nullptr;
  int rc = get_ctx(&c);
  if (rc) return rc;
  const RcSegments g = rc_segments(p, rows, c->sm_count, scratch);
  const unsigned cols = (p.E + RC_E - 1) / RC_E;
  if (g.n > 1) {
    constexpr int smem = (int)SsSmem<DP>::TOTAL;
    static std::atomic<unsigned long long> done{0};
    rc = ensure_dynamic_smem(ssd_state_kernel<DP>, smem, done);
    if (rc) return rc;
    LaunchCfg lc(dim3(cols, p.H, g.n - 1), dim3(RC_THREADS), smem, s, pdl_enabled());
    TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, ssd_state_kernel<DP>, p, (const __nv_bfloat16*)conv, gates, pos0, g));
  }
  constexpr int smem = (int)ScSmem<DP>::TOTAL;
  static std::atomic<unsigned long long> done{0};
  rc = ensure_dynamic_smem(ssd_chunk_kernel<DP>, smem, done);
  if (rc) return rc;
  LaunchCfg lc(dim3(cols, p.H, g.n), dim3(RC_THREADS), smem, s, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, ssd_chunk_kernel<DP>, p, (const __nv_bfloat16*)conv, gates, o, rows, pos0, g));
  return TLB_OK;
}

}  // namespace

bool recur_chunk_eligible(const RecurP& p) { return p.D <= 128 && p.D % 8 == 0 && p.E % 8 == 0 && p.cv.taps <= 8; }

size_t recur_chunk_scratch_bytes(const RecurP& p, int rows) {
  if (p.kind == MIX_DELTA) return (size_t)((rows + RC_L - 1) / RC_L) * p.H * 2 * RC_L * RC_L * 2;
  DeviceCtx* c = nullptr;
  if (get_ctx(&c)) return 0;   // and the launch fails
  const int n = rc_most_segments(p, rows, c->sm_count);
  return n > 1 ? (size_t)n * p.H * ((size_t)p.D * p.E + 1) * sizeof(float) : 0;
}

int recur_chunk_launch(const RecurP& p, const void* conv, const float2* gates, const float2* norms, void* scratch,
                       float* o, int rows, int pos0, cudaStream_t s) {
  if (p.kind == MIX_DELTA)
    return p.D <= 64 ? delta_launch<64>(p, conv, gates, norms, scratch, o, rows, pos0, s)
                     : delta_launch<128>(p, conv, gates, norms, scratch, o, rows, pos0, s);
  return p.D <= 64 ? ssd_launch<64>(p, conv, gates, scratch, o, rows, pos0, s)
                   : ssd_launch<128>(p, conv, gates, scratch, o, rows, pos0, s);
}

}  // namespace tlb
