// int4 dequant-matmul for many activation rows (prefill / batched rows, M > 8; fewer with deep weights), second
// formulation: Y[M,N] = alpha * X[M,K] . dequant(Wq) + beta on the 5th-generation tensor cores
// with the GROUP SCALES KEPT OUT of the tensor-core operands.
//
//   y[m,n] = sum_g sc[n,g] * ( sum_{k in group g} (nib[n,k] - 8) * x[m,k] )
//
// The inner sum is an exact-operand contraction: nib - 8 is an integer in [-8, 7], exact in
// fp16, and x is carried as TWO fp16 planes (hi + lo of x * 2^-e_m, e_m a per-row power of two
// that keeps the row inside the fp16 range; 22 mantissa bits, the precision the tf32 hi/lo
// split gave).  So a group of 32 k costs 2 k-steps x 2 planes = 4 tcgen05.mma.kind::f16
// (K = 16 each) instead of 12 kind::tf32 MMAs at half the rate: a sixth of the tensor time of
// the formulation that folds the f32 scale into the weight operand (gemm_q4_tc.cu), which is
// tensor bound at a third of the tf32 peak.  Each group's product lands in one of four TMEM
// accumulators (three at 128 columns) used in rotation; accumulate warps read it back with tcgen05.ld, multiply by
// the row's f32 group scale and add into registers -- the same order of operations as the
// reference's dequantise-then-multiply in f32 (include/array.h:666-684, 1980-1984).
//
// A tile is 128 weight rows (UMMA M) x MT activation rows (UMMA N, 32 / 64 / 128); its work is a row of units of
// 256 k (one box of packed weights).  The CTAs, one per SM at most, stay for the whole product and take equal
// ranges of the units, tile after tile: the pipelines below run on across the tiles, so that a tile's first loads and
// conversions pass under the stores of the one before, and a product with few tiles still uses the
// whole chip.  A tile whose units lie in several CTAs' ranges is summed by the last of them to finish, in
// the order of k, from f32 partials in scratch (T2Work): the same bits on every call, and no CTA waits for
// another.  Warp roles (512 threads): warp 0 TMA producer of the X planes (64-k stages, 128-byte swizzle), warp 1 TMEM
// allocator, warps 1 and 2 the MMA issuers (first / second group of a stage), warp 3 TMA producer of the PACKED weights
// (128 rows x 128 bytes = 256 k a box, a ring of four: 64 KB in flight an SM), warps 4-7 nibble -> fp16 converters (thread r
// owns weight row r; the k order inside every group of 8 is the one the nibble extraction produces -- 0,4,1,5,2,6,3,7 -- and
// the X planes are stored in the same order, so no byte permute is needed), warps 8-15 accumulate + epilogue (two per TMEM
// lane quarter, each half of the MT columns).  The converters leave the weights in TMEM, a lane a row: the A operand of the
// MMAs comes from there.  At 128 columns the feeding warpgroups give registers to the accumulating ones.  All waits are bounded; a timeout
// sets the status word, the kernel still frees its TMEM and returns, and no warp is split by it.  No cluster launch, no
// multicast.
//
// What bounds it: at large sizes the power limit (1620 MHz of 1965 at 1000 x 3584 x 37888), and at all sizes the way of an
// accumulator from its MMAs to the accumulate warps and back.  Per group of 32 k and 128 columns the tensor pipe works 256
// cycles; an issuer takes about 600 (61 an MMA to issue, 130 the look at its barriers, 70 the commits), so there are two; an
// accumulate warp 90 to read 64 columns and about 270 for the FMAs that it shares a scheduler with.  What was done about it,
// 1000 x 3584 x 37888 / 517 x 896 x 9728 in one loop of products, us: 656 / 38.4 before; all of a warp's columns in one read
// into registers that setmaxnreg gives it, the accumulator back before the FMAs; one barrier for a stage's two operands and
// one vote an issuer's group; the look at the next group's barrier under the FMAs; weights in TMEM, which takes 32 of 120 KB
// a stage off the shared memory; the odd nibbles of a byte converted in place by one FMA: 611 / 34.9.  Measured beside it: two
// sets of accumulate warps that take the groups in turn (588 against 579 of that time), four stages of operands (no change),
// one issuer (551 against 517) or three (615 against 611), the next read under a group's FMAs (634), pairs of columns by
// fma.rn.f32x2 at 128 columns (632), sixteen accumulate warps, leaving out the reads of columns behind the last row.
#include <cstdlib>

#include "q4_planes.cuh"

namespace tlb {

namespace {

constexpr int T2_THREADS = 512;
constexpr int T2_ROWS = 128;     // weight rows per CTA (UMMA M)
constexpr int T2_KS = 64;        // k per stage = two groups = one 128-byte swizzle row of fp16
constexpr int T2_RAW_BYTES = T2_ROWS * 128;   // one box: 128 rows x 128 bytes = 256 k per row
constexpr int T2_SUB = 4;                     // 64-k stages per packed box
// Registers a thread of the two warpgroups that feed the tensor pipe, and of the two that accumulate: 256 (72 + 184) =
// what 512 threads of 128 are launched with.  At 128 columns alone: up to 64 the accumulators fit 108 registers a thread, and
// what that leaves of an SM's takes the first blocks of the next launch (the split of its rows).  Products on all SMs, one
// behind the other, us with the exchange / without: 64 x 3584 x 3584 19.3 / 17.5, 16 rows 16.2 / 14.5, 64 x 3584 x 4608
// 20.0 / 18.2; where the split takes 1024 threads a row, or SMs are idle anyway, nothing (64 x 18944 x 3584 38.0 / 38.2).
constexpr int T2_REGS_FEED = 72, T2_REGS_ACC = 184;

struct T2Params {
  const unsigned* qw;        // packed nibbles, u32 [N][K/8]
  const float* scales;       // [N][K/32]
  const float* rowscale;     // [M] 2^e_m
  float* y;
  long long ldy;
  int M, N, K;
  float alpha, beta;
  int* status;
  int n_tiles, box;          // tiles along N (the inner ones), units of a tile
  unsigned per, longer, grain;   // units a CTA / grain, CTAs with one more, grain = 1 or box (whole tiles)
  float* parts;              // [2 * CTAs][MT][128]
  int* tickets;              // [CTAs], zero between launches
};

// Which units are a CTA's: ranges of `per` or per + 1 units (or whole tiles), the tiles in order.
__device__ __forceinline__ unsigned t2_first(const T2Params& p, unsigned cta) {
  return (cta * p.per + (cta < p.longer ? cta : p.longer)) * p.grain;
}
// the CTA whose range holds unit u
__device__ __forceinline__ unsigned t2_owner(const T2Params& p, unsigned u) {
  const unsigned v = u / p.grain, in_longer = p.longer * (p.per + 1);
  return v < in_longer ? v / (p.per + 1) : p.longer + (v - in_longer) / p.per;
}
// The CTA's segments in order: boxes q0 .. q1 of a tile.
struct T2Segment {
  unsigned u, end;
  int tile = 0, q0 = 0, q1 = 0;
  __device__ __forceinline__ T2Segment(const T2Params& p) : u(t2_first(p, blockIdx.x)), end(t2_first(p, blockIdx.x + 1)) {}
  __device__ __forceinline__ bool next(const T2Params& p) {
    if (u >= end) return false;
    tile = (int)(u / (unsigned)p.box);
    q0 = (int)(u - (unsigned)tile * (unsigned)p.box);
    q1 = (unsigned)(p.box - q0) < end - u ? p.box : q0 + (int)(end - u);
    u += (unsigned)(q1 - q0);
    return true;
  }
};

template <int MT>
struct T2Smem {
  static constexpr int STAGES = 4, RAW_STAGES = 4;                            // rings of operands, of weight boxes
  static constexpr size_t B = 0;                                              // [stages][2 planes][MT][128 B]
  static constexpr size_t RAW = B + (size_t)STAGES * 2 * MT * 128;            // [raw stages][128][128 B]
  static constexpr size_t BARS = RAW + (size_t)RAW_STAGES * T2_RAW_BYTES;
  static constexpr size_t SLOT = BARS + 32 * 8;
  static constexpr size_t TOTAL = SLOT + 16 + 1024;
};

__device__ __forceinline__ void t2_alloc(uint32_t* slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void t2_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void t2_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void t2_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t2_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t2_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// A from TMEM (a lane a row, two k a column), B from shared memory
__device__ __forceinline__ void t2_mma_f16(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 lanes x 16 consecutive columns of this warp's TMEM lane quarter (issue only; see t2_wait_ld)
__device__ __forceinline__ void t2_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 32 consecutive columns of this warp's TMEM lane quarter, written and there when it returns
__device__ __forceinline__ void t2_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// two f32 FMAs an instruction: c + (s, s) * (a, b)
__device__ __forceinline__ void t2_fma2(unsigned long long& c, unsigned long long s2, uint32_t a, uint32_t b) {
  asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%2, %3};\n\tfma.rn.f32x2 %0, %1, v, %0;\n\t}" : "+l"(c) : "l"(s2), "r"(a), "r"(b));
}
__device__ __forceinline__ bool t2_elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
// The converters' wait: no outcome to branch on.  A wait that gives up marks the CTA, the converters then wait no more
// but stay together to the end, and the epilogue writes nothing.
__device__ __forceinline__ void t2_wait_or_mark(uint64_t* bar, uint32_t parity, int* status, int where,
                                                volatile int* gave_up) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (clock64() - t0 < 8192)   // see mbar_wait_bounded
    if (mbar_try_wait(bar, parity)) return;
  const long long limit = wait_limit(status);
  while (!*gave_up) {
    if (mbar_try_wait(bar, parity)) return;
    if (clock64() - t0 > limit) {
      *gave_up = 1;
      if (status) {
        atomicExch(&status[ST_WAIT_TIMEOUT], 1);
        atomicExch(&status[ST_WAIT_WHERE], where);
      }
    }
  }
}
// a look at a barrier that never suspends the warp
__device__ __forceinline__ bool t2_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void t2_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major, 128-byte swizzle shared-memory matrix descriptor: rows of 128 bytes, 8-row groups
// 1024 bytes apart (the layout TMA's SWIZZLE_128B box produces and the converters write).
__device__ __forceinline__ uint64_t t2_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16 with fp16 operands (format code 0), f32 accumulate, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t t2_idesc_f16(int n) {
  uint32_t d = 0;
  d |= 1u << 4;                          // D format f32
  d |= (uint32_t)(n >> 3) << 17;         // N / 8
  d |= (uint32_t)(T2_ROWS >> 4) << 24;   // M / 16
  return d;
}

// barrier indices
enum { T2_ST_FULL = 0, T2_ST_EMPTY = 8, T2_D_FULL = 12, T2_D_EMPTY = 16, T2_RAW_FULL = 20,
       T2_RAW_EMPTY = 24 };
// TMEM accumulators in rotation: the issuers run up to that many groups ahead of the accumulate warps.  The rest of
// TMEM holds the stages' weights.
constexpr int t2_nbuf(int mt) { return mt == 128 ? 3 : 4; }
constexpr int T2_A_COLS = T2_KS / 2;   // TMEM columns of a stage's weights

template <int MT>
__global__ void __launch_bounds__(T2_THREADS, 1)
    gemm_q4_tc2_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                       const __grid_constant__ CUtensorMap tmW, T2Params p) {
  using S = T2Smem<MT>;
  constexpr int T2_STAGES = S::STAGES, T2_RAW_STAGES = S::RAW_STAGES;
  constexpr int T2_NBUF = t2_nbuf(MT);
  constexpr uint32_t A_AT = T2_NBUF * MT;    // TMEM: accumulators of MT columns each, then the weights
  constexpr uint32_t NCOLS = MT == 32 ? 256 : 512;
  static_assert(A_AT + T2_STAGES * T2_A_COLS <= NCOLS, "TMEM");
  constexpr int HC = MT / 2;              // columns per accumulate warp
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = (uint64_t*)(base + S::BARS);
  uint32_t* tmem_slot = (uint32_t*)(base + S::SLOT);
  volatile int *last_part = (volatile int*)(base + S::SLOT + 8), *gave_up = last_part + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = p.K / T2_KS;   // 64-k stages of a tile
  T2Segment sg(p);

  if (tid == 0) {
    *gave_up = 0;
    for (int s = 0; s < T2_STAGES; s++) {
      mbar_init(&bars[T2_ST_FULL + s], 5);    // the X planes' copy, four converter warps
      mbar_init(&bars[T2_ST_EMPTY + s], 2);   // one commit per issuer warp
    }
    for (int b = 0; b < T2_NBUF; b++) {
      mbar_init(&bars[T2_D_FULL + b], 1);
      mbar_init(&bars[T2_D_EMPTY + b], 8);
    }
    for (int q = 0; q < T2_RAW_STAGES; q++) {
      mbar_init(&bars[T2_RAW_FULL + q], 1);
      mbar_init(&bars[T2_RAW_EMPTY + q], 4);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    t2_alloc(tmem_slot, NCOLS);
    t2_relinquish();
  }
  t2_fence_before();
  __syncthreads();
  t2_fence_after();
  const uint32_t tmem = *tmem_slot;

  // the packed weights are not written by the kernel before this one: their producer starts
  // at once; every other role touches activations, the status block or y and waits
  if (warp != 3) pdl_wait();
  pdl_launch_dependents();

  if (warp < 8) {
    if constexpr (MT == 128) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(T2_REGS_FEED));
  if (warp == 3) {
    // ---------------- TMA producer: packed weights, 128 rows x 256 k per box ----------------
    if (lane == 0) {
      int cnt = 0;
      bool ok = true;
      while (sg.next(p)) {
        const int n0 = sg.tile % p.n_tiles * T2_ROWS;
        for (int q = sg.q0; q < sg.q1 && ok; q++, cnt++) {
          const int rs = cnt % T2_RAW_STAGES;
          ok = mbar_wait_bounded(&bars[T2_RAW_EMPTY + rs], ((cnt / T2_RAW_STAGES) & 1) ^ 1, p.status, 640);
          if (!ok) break;
          mbar_expect_tx(&bars[T2_RAW_FULL + rs], (uint32_t)T2_RAW_BYTES);
          tma_load_2d(base + S::RAW + (size_t)rs * T2_RAW_BYTES, &tmW, q * 128, n0, &bars[T2_RAW_FULL + rs]);
        }
      }
    }
  } else if (warp == 0) {
    // ---------------- TMA producer: the two fp16 planes of X, one 64-k stage at a time ----------------
    if (lane == 0) {
      int cnt = 0;
      bool ok = true;
      while (sg.next(p)) {
        const int m0 = sg.tile / p.n_tiles * MT, it1 = sg.q1 * T2_SUB < nst ? sg.q1 * T2_SUB : nst;
        for (int it = sg.q0 * T2_SUB; it < it1 && ok; it++, cnt++) {
          const int s = cnt % T2_STAGES;
          ok = mbar_wait_bounded(&bars[T2_ST_EMPTY + s], ((cnt / T2_STAGES) & 1) ^ 1, p.status, 600);
          if (!ok) break;
          mbar_expect_tx(&bars[T2_ST_FULL + s], 2u * MT * 128u);
          const int kx = it * T2_KS;
          tma_load_2d(base + S::B + (size_t)(s * 2 + 0) * MT * 128, &tmX1, kx, m0, &bars[T2_ST_FULL + s]);
          tma_load_2d(base + S::B + (size_t)(s * 2 + 1) * MT * 128, &tmX2, kx, m0, &bars[T2_ST_FULL + s]);
        }
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ---------------- MMA issuers: warp 1 the first group of every stage, warp 2 the second ----------------
    // The whole warp runs the loop (waits included) so that descriptors and addresses stay
    // warp-uniform values, and one elected lane issues; two issuers because the issue cost of
    // a tcgen05.mma (not its execution) bounds a single thread at this instruction size.
    const int grp = warp == 1 ? 0 : 1;
    const uint32_t idesc = t2_idesc_f16(MT);
    const bool leader = t2_elect_one();
    int stages = 0;   // of all segments: tiles follow one another without a seam
    while (sg.next(p)) stages += (sg.q1 * T2_SUB < nst ? sg.q1 * T2_SUB : nst) - sg.q0 * T2_SUB;
    for (int it = 0; it < stages; it++) {
      const int s = it % T2_STAGES;
      const uint32_t ph = (it / T2_STAGES) & 1;
      const int gi = 2 * it + grp, buf = gi % T2_NBUF;
      // one vote for both barriers where they are complete on the first look
      const uint32_t dph = ((gi / T2_NBUF) & 1) ^ 1;
      const bool there = mbar_try_wait(&bars[T2_ST_FULL + s], ph) & mbar_try_wait(&bars[T2_D_EMPTY + buf], dph);
      if (!__all_sync(0xffffffffu, there)) {
        if (!mbar_wait_warp(&bars[T2_D_EMPTY + buf], dph, p.status, 612)) break;
        if (!mbar_wait_warp(&bars[T2_ST_FULL + s], ph, p.status, 610)) break;
      }
      t2_fence_after();
      const uint32_t a = tmem + A_AT + (uint32_t)(s * T2_A_COLS);
      const uint64_t b1 = t2_desc_sw128(smem_u32(base + S::B + (size_t)(s * 2 + 0) * MT * 128));
      const uint64_t b2 = t2_desc_sw128(smem_u32(base + S::B + (size_t)(s * 2 + 1) * MT * 128));
      const uint32_t d = tmem + (uint32_t)(buf * MT);
      if (leader) {
#pragma unroll
        for (int ks = 0; ks < 2; ks++) {
          const uint64_t adv = (uint64_t)(((2 * grp + ks) * 32) >> 4);   // 16 fp16 = 32 bytes along K
          const uint32_t ak = a + (uint32_t)((2 * grp + ks) * 8);        // or 8 columns
          t2_mma_f16(d, ak, b1 + adv, idesc, ks ? 1u : 0u);
          t2_mma_f16(d, ak, b2 + adv, idesc, 1u);
        }
        t2_commit(&bars[T2_D_FULL + buf]);     // the group's product is complete when these retire
        t2_commit(&bars[T2_ST_EMPTY + s]);     // ... and (with the other issuer's) the stage can be overwritten
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ---------------- nibble -> fp16 converters (thread r = weight row r) ----------------
    const int r = tid - 128;
    const __half2 off = __floats2half2_rn(1032.0f, 1032.0f), odd = __floats2half2_rn(0.0625f, 0.0625f),
                  odd_off = __floats2half2_rn(-72.0f, -72.0f);
    int cnt = 0, it = -1;   // boxes and stages of all segments
    while (sg.next(p)) for (int q = sg.q0; q < sg.q1; q++, cnt++) {
      const int rs = cnt % T2_RAW_STAGES;
      t2_wait_or_mark(&bars[T2_RAW_FULL + rs], (cnt / T2_RAW_STAGES) & 1, p.status, 621, gave_up);
      // the row's 128 packed bytes of this box: chunk c (16 bytes = 32 k) sits at c ^ (r & 7)
      const unsigned char* rrow = base + S::RAW + (size_t)rs * T2_RAW_BYTES + r * 128;
#pragma unroll 1
      for (int u = 0; u < T2_SUB; u++) {
        if (q * T2_SUB + u >= nst) break;
        it++;
        const int s = it % T2_STAGES;
        const uint4 c0 = *(const uint4*)(rrow + (((2 * u) ^ (r & 7)) << 4));
        const uint4 c1 = *(const uint4*)(rrow + (((2 * u + 1) ^ (r & 7)) << 4));
        t2_wait_or_mark(&bars[T2_ST_EMPTY + s], ((it / T2_STAGES) & 1) ^ 1, p.status, 620, gave_up);
        uint32_t qv[32];
        const unsigned words[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int j = 0; j < 8; j++) {
          // slot e of the chunk holds (k = e, k = e + 4) of this word: fp16(1024 + nib) has the
          // bit pattern 0x6400 | nib, and 1024 + nib - 1032 = nib - 8 exactly
          // (and the odd nibbles of a byte in place: (1024 + 16 nib) / 16 - 72)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const unsigned w = words[j] >> (8 * e), t = (w & 0x000F000Fu) | 0x64006400u, o = (w & 0x00F000F0u) | 0x64006400u;
            const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&t), off);
            const __half2 z = __hfma2(*reinterpret_cast<const __half2*>(&o), odd, odd_off);
            qv[4 * j + 2 * e] = *reinterpret_cast<const unsigned*>(&v);
            qv[4 * j + 2 * e + 1] = *reinterpret_cast<const unsigned*>(&z);
          }
        }
        t2_fence_after();
        t2_st32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + A_AT + (uint32_t)(s * T2_A_COLS), qv);
        t2_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[T2_ST_FULL + s]);
      }
      // The box goes back only here, behind the stores that used all of it.  Given back right after the
      // loads above (which need not be complete, or even issued, before their first use) it was refilled under its readers:
      // 60 of 60 products with M = 32, K = 3584, N = 18944 had wrong rows.
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[T2_RAW_EMPTY + rs]);
    }
  }
  } else {
    // ---------------- accumulate (sc * group product) + epilogue ----------------
    if constexpr (MT == 128) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(T2_REGS_ACC));
    const int quarter = warp & 3, half = (warp - 8) >> 2;
    const int r = quarter * 32 + lane;
    const int c_lo = half * HC;
    bool ok = true;   // of the warp.  A wait that gave up: no more work, but every barrier and ticket below
    int buf = 0;           // accumulator of the next group
    unsigned parity = 0;
    bool there = false;    // the next group is known to be complete
    while (sg.next(p)) {
      const int tile = sg.tile, q0 = sg.q0, q1 = sg.q1;
      const int n = tile % p.n_tiles * T2_ROWS + r, m0 = tile / p.n_tiles * MT;
      // 32 and 64 columns: in pairs of columns, two FMAs an instruction (64 x 3584 x 18944 31.9 -> 28.9 us, 16 rows 27.7 ->
      // 26.2); at 128 columns that loses (610 -> 634 us)
      constexpr bool PAIRS = MT < 128;
      float acc[HC];
      unsigned long long acc2[PAIRS ? HC / 2 : 1];
#pragma unroll
      for (int i = 0; i < HC; i++) {
        acc[i] = 0.f;
        if (PAIRS) acc2[PAIRS ? i / 2 : 0] = 0ull;
      }
      // the row's group scales, four at a time (K % 128 == 0), fetched a block ahead: an L2 round trip is
      // shorter than the four groups take
      const float4* sc4 = (const float4*)(p.scales + (size_t)(n < p.N ? n : p.N - 1) * (p.K / 32)) + q0 * 2;
      const int nblk = (q1 * 2 < p.K / 128 ? q1 * 2 : p.K / 128) - q0 * 2;
      float4 sc_blk = __ldg(sc4);
      for (int b = 0; b < nblk && ok; b++) {
        const float4 sc_next = b + 1 < nblk ? __ldg(sc4 + b + 1) : sc_blk;
#pragma unroll
        for (int k = 0; k < 4; k++) {   // four groups a block
          const float sc = k == 0 ? sc_blk.x : (k == 1 ? sc_blk.y : (k == 2 ? sc_blk.z : sc_blk.w));
          if (!__all_sync(0xffffffffu, there) && !mbar_wait_warp(&bars[T2_D_FULL + buf], parity, p.status, 630)) {
            ok = false;
            break;
          }
          t2_fence_after();
          const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * MT + c_lo);
          // All of the warp's columns in one read: the accumulator goes back to the issuers as soon as it has landed, before
          // the FMAs, and the look at the next group's barrier passes under them.
          uint32_t v[HC / 16][16];
#pragma unroll
          for (int i = 0; i < HC / 16; i++) t2_ld16_issue(taddr + (uint32_t)(16 * i), v[i]);
          t2_wait_ld();
          t2_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[T2_D_EMPTY + buf]);
          if (++buf == T2_NBUF) { buf = 0; parity ^= 1u; }
          there = t2_test(&bars[T2_D_FULL + buf], parity);
          if constexpr (PAIRS) {
            unsigned long long sc2;
            asm("mov.b64 %0, {%1, %1};" : "=l"(sc2) : "f"(sc));
#pragma unroll
            for (int i = 0; i < HC; i += 2) t2_fma2(acc2[i / 2], sc2, v[i / 16][i % 16], v[i / 16][i % 16 + 1]);
          } else {
#pragma unroll
            for (int i = 0; i < HC; i++) acc[i] = fmaf(sc, __uint_as_float(v[i / 16][i % 16]), acc[i]);
          }
        }
        sc_blk = sc_next;
      }
      if constexpr (PAIRS)
#pragma unroll
        for (int i = 0; i < HC / 2; i++) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[2 * i]), "=f"(acc[2 * i + 1]) : "l"(acc2[i]));
      bool mine = true;   // this CTA writes the tile
      if (q1 - q0 < p.box) {
        // a part of the tile: into scratch, and the last of the tile's CTAs sums all parts
        const unsigned u0 = (unsigned)tile * (unsigned)p.box;
        const int first = (int)t2_owner(p, u0), last = (int)t2_owner(p, u0 + (unsigned)p.box - 1u), me = blockIdx.x;
        auto part = [&](int cta) {
          const int second = t2_first(p, cta) < u0;   // the range began in an earlier tile
          return p.parts + (size_t)(2 * cta + second) * (MT * T2_ROWS) + (size_t)c_lo * T2_ROWS + r;
        };
        float* mp = part(me);
#pragma unroll
        for (int i = 0; i < HC; i++) __stcg(mp + i * T2_ROWS, acc[i]);
        __threadfence();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (warp == 8 && lane == 0) {
          int old;
          asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(p.tickets + first) : "memory");
          *last_part = old == last - first;
          if (old == last - first) p.tickets[first] = 0;   // clean for the next launch
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        mine = *last_part != 0;
        if (mine) {
#pragma unroll
          for (int i = 0; i < HC; i++) acc[i] = 0.f;
          for (int cta = first; cta <= last; cta++) {
            const float* q = part(cta);
#pragma unroll
            for (int i = 0; i < HC; i++) acc[i] += __ldcg(q + i * T2_ROWS);
          }
        }
      }
      if (mine && ok && !*gave_up && n < p.N) {
#pragma unroll
        for (int i = 0; i < HC; i++) {
          const int m = m0 + c_lo + i;
          if (m < p.M) p.y[(long long)m * p.ldy + n] = (acc[i] * __ldg(p.rowscale + m)) * p.alpha + p.beta;
        }
      }
      __syncwarp();   // lanes of rows behind the last: whole warps again for the next segment's reads
    }
  }
  t2_fence_before();
  __syncthreads();
  if (warp == 1) {
    t2_fence_after();
    t2_dealloc(tmem, NCOLS);
  }
}

// X -> two fp16 planes of x * 2^-e_m (hi, lo) + the row's 2^e_m.  One block per row.  Inside every
// group of 8 k the planes are stored in the order 0,4,1,5,2,6,3,7 -- the order in which the
// converters' nibble extraction lays out the weights.
constexpr int SPLIT_MOST = 1024;   // threads a row
__global__ void __launch_bounds__(SPLIT_MOST)
    split_f16_kernel(const float* __restrict__ x, long long ldx, int K, __half* __restrict__ x1, __half* __restrict__ x2,
                     float* __restrict__ rowscale) {
  __shared__ float sm[32];
  pdl_wait();
  pdl_launch_dependents();
  const int m = blockIdx.x;
  const float* row = x + (long long)m * ldx;
  const bool vec = ((uintptr_t)row & 15) == 0;   // K % 8 == 0 always; 16-byte rows take the float4 path
  float mx = 0.f;
  if (vec) {
    const float4* row4 = (const float4*)row;
    for (int i = threadIdx.x; i < K / 4; i += blockDim.x) {
      const float4 a = __ldg(row4 + i);
      mx = fmaxf(fmaxf(mx, fmaxf(fabsf(a.x), fabsf(a.y))), fmaxf(fabsf(a.z), fabsf(a.w)));
    }
  } else {
    for (int k = threadIdx.x; k < K; k += blockDim.x) mx = fmaxf(mx, fabsf(row[k]));
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) mx = fmaxf(mx, sm[w]);
  const int e = q4_row_exponent(mx);
  const float s = ldexpf(1.0f, -e);
  if (threadIdx.x == 0) rowscale[m] = ldexpf(1.0f, e);
  if (vec) {
    const float4* row4 = (const float4*)row;
    uint4* o1 = (uint4*)(x1 + (size_t)m * K);
    uint4* o2 = (uint4*)(x2 + (size_t)m * K);
    for (int i = threadIdx.x; i < K / 8; i += blockDim.x) {
      const float4 a = __ldg(row4 + 2 * i), b = __ldg(row4 + 2 * i + 1);
      uint4 w1, w2;
      q4_split8(a, b, s, w1, w2);
      o1[i] = w1;
      o2[i] = w2;
    }
    return;
  }
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float v = row[k] * s;
    const __half h1 = __float2half_rn(v);
    const __half h2 = __float2half_rn(v - __half2float(h1));
    const int k8 = k & 7;
    const size_t pos = (size_t)m * K + (k & ~7) + (k8 < 4 ? 2 * k8 : 2 * (k8 - 4) + 1);
    x1[pos] = h1;
    x2[pos] = h2;
  }
}

template <int MT>
int t2_launch(const CUtensorMap& tm1, const CUtensorMap& tm2, const CUtensorMap& tmw, const T2Params& p,
              int ctas, cudaStream_t stream) {
  static std::atomic<unsigned long long> attr_done{0};
  {
    const int rc_attr = ensure_dynamic_smem(gemm_q4_tc2_kernel<MT>, (int)T2Smem<MT>::TOTAL, attr_done);
    if (rc_attr) return rc_attr;
  }
  LaunchCfg lc(dim3(ctas), dim3(T2_THREADS), T2Smem<MT>::TOTAL, stream, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, gemm_q4_tc2_kernel<MT>, tm1, tm2, tmw, p));
  return TLB_OK;
}

}  // namespace

// tickets (zeroed once by the owner) and parts of the tiles that several CTAs share
size_t gemm_q4_work_bytes(int sm_count) { return Q4_TICKET_BYTES + (size_t)2 * sm_count * 128 * T2_ROWS * sizeof(float); }

// bytes of the activation scratch: two fp16 planes + the row scales
size_t gemm_q4_tc2_scratch_bytes(int M, int K) { return (size_t)M * K * 4 + (size_t)((M + 3) & ~3) * 4 + 256; }

bool gemm_q4_tc2_eligible(const void* qw, const void* scales, int N, int K, int M) {
  if (M <= 0 || N <= 0 || M > 65535 * 32) return false;
  if (K % 128 != 0) return false;
  return (((uintptr_t)qw & 15) == 0) && (((uintptr_t)scales & 15) == 0);
}

bool gemm_q4_planes_eligible(const void* qw, const void* scales, int N, int K, int M) {
  return M > 8 && gemm_q4_planes_possible(qw, scales, N, K, M);
}

bool gemm_q4_planes_possible(const void* qw, const void* scales, int N, int K, int M) {
  // TLB_GEMM_TC=1 selects the earlier formulation (gemm_q4_tc.cu)
  static const bool tc_old = getenv("TLB_GEMM_TC") && atoi(getenv("TLB_GEMM_TC")) == 1;
  return !tc_old && gemm_q4_tc2_eligible(qw, scales, N, K, M);
}

int gemm_q4_tc2_launch(DeviceCtx* c, const float* x, long long ldx, int M, const void* qw, const float* scales,
                       float* y, long long ldy, int N, int K, float alpha, float beta, void* scratch,
                       void* work, cudaStream_t stream) {
  const Q4Planes pl = q4_planes_at(scratch, M, K);
  const int rc = launch_split_rows(x, ldx, M, K, pl, c->sm_count, stream);
  return rc ? rc : gemm_q4_planes_launch(c, pl, M, qw, scales, y, ldy, N, K, alpha, beta, work, stream);
}

int launch_split_rows(const float* x, long long ldx, int M, int K, const Q4Planes& pl, int sms, cudaStream_t stream) {
  // few deep rows: more threads a row, since there are fewer rows than SMs (8 x 18944, split and product: 41.8 -> 32.5 us)
  const int threads = M <= sms && K >= 4096 ? SPLIT_MOST : 256;
  LaunchCfg lc(dim3((unsigned)M), dim3(threads), 0, stream, pdl_enabled());
  TLB_CUDA(cudaLaunchKernelEx(&lc.cfg, split_f16_kernel, x, ldx, K, pl.hi, pl.lo, pl.rowscale));
  return TLB_OK;
}

int gemm_q4_planes_launch(DeviceCtx* c, const Q4Planes& x, int M, const void* qw, const float* scales, float* y,
                          long long ldy, int N, int K, float alpha, float beta, void* work, cudaStream_t stream) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return set_error(TLB_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
  const int MT = M <= 32 ? 32 : (M <= 64 ? 64 : 128);
  CUtensorMap tm1, tm2;
  cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)M};
  cuuint64_t str[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)T2_KS, (cuuint32_t)MT};
  cuuint32_t es[2] = {1, 1};
  if (enc(&tm1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x.hi, dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
          CUDA_SUCCESS ||
      enc(&tm2, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x.lo, dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
          CUDA_SUCCESS)
    return set_error(TLB_ERR_CUDA, "gemm_q4_tc2: tensor map (activation planes) encode failed");
  // packed weights as bytes [N][K/2]; boxes past K/2 or N read as zeros and are never converted / stored
  CUtensorMap tmw;
  cuuint64_t wdim[2] = {(cuuint64_t)K / 2, (cuuint64_t)N};
  cuuint64_t wstr[1] = {(cuuint64_t)K / 2};
  cuuint32_t wbox[2] = {128, (cuuint32_t)T2_ROWS};
  if (enc(&tmw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(qw), wdim, wstr, wbox, es,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return set_error(TLB_ERR_CUDA, "gemm_q4_tc2: tensor map (packed weights) encode failed");
  T2Params p;
  p.qw = (const unsigned*)qw; p.scales = scales; p.rowscale = x.rowscale; p.y = y; p.ldy = ldy;
  p.M = M; p.N = N; p.K = K; p.alpha = alpha; p.beta = beta; p.status = c->status;
  p.n_tiles = (N + T2_ROWS - 1) / T2_ROWS;
  p.box = (K / T2_KS + T2_SUB - 1) / T2_SUB;
  p.tickets = (int*)work;
  p.parts = (float*)((char*)work + Q4_TICKET_BYTES);
  // Whole tiles for each CTA, or equal ranges of units (no tile in more than eight or so) where what the last,
  // partly empty round of tiles would leave idle is worth more than writing and reading the parts: from four units of
  // 256 k an SM on.  517 x 896 x 9728 (1.7 units idle) takes 46 us in tiles and 51 in ranges, 64 x 3584 x 3584
  // (11 idle) 34 in tiles and 24 in ranges, 1000 x 3584 x 3584 (6.8 idle) 93 and 85.
  const long long tiles = (long long)p.n_tiles * ((M + MT - 1) / MT), sms = c->sm_count, units = tiles * p.box;
  if (units >= 1ll << 31) return set_error(TLB_ERR_UNSUPPORTED, "gemm_q4: 2^31 units of 256 k or more");
  const long long rounds = (tiles + sms - 1) / sms, idle = (rounds * sms - tiles) * p.box;   // in units
  const bool split = idle >= 4 * sms;
  const long long least = (p.box + 7) / 8;
  const long long grains = split ? units : tiles;
  long long ctas = split ? units / least : tiles;
  if (ctas > sms) ctas = sms;
  p.grain = split ? 1 : (unsigned)p.box;
  p.per = (unsigned)(grains / ctas);
  p.longer = (unsigned)(grains % ctas);
  if (MT == 32) return t2_launch<32>(tm1, tm2, tmw, p, (int)ctas, stream);
  if (MT == 64) return t2_launch<64>(tm1, tm2, tmw, p, (int)ctas, stream);
  return t2_launch<128>(tm1, tm2, tmw, p, (int)ctas, stream);
}

}  // namespace tlb
