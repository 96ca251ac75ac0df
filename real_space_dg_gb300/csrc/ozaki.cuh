// FP64 GEMM emulated on the BF16 tensor cores (Ozaki splitting), sm_103a.
//
//   C (M x Ncol, fp64, column-major)  (=|+=)  A (M x K, fp64)  *  B (K x Ncol, fp64, column-major)
//
// Each row of A and each column of B is scaled by a power of two and rounded to
// an integer F with |F| <= 2^(6S-1), which is written in S balanced base-64
// digits: a = 2^e sum_p t_p 2^(-6(p+1)), |t_p| <= 32 (|t_0| <= 33).  The digits
// are exact in BF16 and a digit product summed over K <= 1024 stays below
// 33^2 * 1024 < 2^21, so every product A^(p) B^(q) is EXACT in the FP32 tensor-core
// accumulator.  Products of equal weight p+q (at most 8 of them) share one TMEM
// accumulator (< 8 * 33^2 * 1024 < 2^24, still exact); the S groups of a 128 x 64 output tile use 8 x 64 = 512
// TMEM columns.  Products of weight p+q >= S are dropped.  The B digit slices lie
// one after the other in shared memory, so the products of one A slice p with the
// slices q = q0 .. q0+n-1 are ONE instruction of N = 64 n (n <= 4) whose accumulator
// starts at group p+q0: 12 MMAs per k step instead of 36, and the A tile is read
// from shared memory 12 times instead of 36.  The epilogue adds the groups as
// integers in a 64-bit fixed point (unit 2^-50), rounds once to FP64 and applies
// the row and column exponents, all with integer instructions.  Error: a few
// 2^(-6S) (S = 8: ~1e-14) relative to |A| |B|, unbiased (rounded split).
#pragma once
#include "tc_gemm.cuh"

namespace wg {
namespace oz {

constexpr int S = 8;              // digits per operand
constexpr int BETA = 6;           // bits per digit
// k blocks of 32 (64-byte rows, 64-byte swizzle).  A stage holds the nd A and nd B slices
// the launch uses, so the 192 KiB ring has two stages at 7 or 8 digits and more with fewer
// digits (three at 5, four at 4): the TMA loads run further ahead of the MMAs
constexpr int BM = 128, BN = 64, BK = 32, STAGES = 2, MAX_STAGES = 8;
constexpr int THREADS = 512;      // warp 0 TMA, warp 1 MMA, all 16 drain TMEM (four warps per lane quarter)
constexpr int EPI_COLS = BN / (THREADS / 128);   // 16 output columns per epilogue warp
static_assert(EPI_COLS == 16, "the epilogue drains 16 TMEM columns per warp");
constexpr int NGROUP = S;         // weights p+q = 2 .. S+1
constexpr int A_SLICE = BM * BK * 2;      // 8 KiB
constexpr int B_SLICE = BN * BK * 2;      // 4 KiB
constexpr int STAGE = S * (A_SLICE + B_SLICE);   // 96 KiB (all 8 digits)
constexpr int RING = STAGES * STAGE;              // 192 KiB
constexpr int SMEM_BYTES = RING + 1024 + 256;
__host__ __device__ constexpr int stages_for(int nd) {
  return RING / (nd * (A_SLICE + B_SLICE)) < MAX_STAGES ? RING / (nd * (A_SLICE + B_SLICE)) : MAX_STAGES;
}
constexpr int MAX_K = 1024;       // exactness bound of the grouped accumulation (8 * 33^2 * K < 2^24)

// Instruction descriptor: D f32, A/B bf16, K-major, M = 128, N = n (16 <= n <= 256, n % 16 == 0).
constexpr uint32_t kIdescM128 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BM >> 4) << 24);
__device__ __forceinline__ uint32_t idesc_n(int n) { return kIdescM128 | ((uint32_t)(n >> 3) << 17); }
constexpr int kSlicesPerMma = 256 / BN;   // B slices one instruction covers (N <= 256)

// K-major operand tile with 64-byte rows and the 64-byte swizzle (8-row atoms of 512 bytes).
__device__ __forceinline__ uint64_t sdesc_sw64(const void* p) {
  const uint64_t addr = tc::smem_u32(p);
  uint64_t d = 0;
  d |= (addr >> 4) & 0x3FFFull;
  d |= 1ull << 16;                    // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;    // stride byte offset: 8 rows x 64 bytes
  d |= 1ull << 46;                    // descriptor version
  d |= 4ull << 61;                    // 64-byte swizzle
  return d;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(tc::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(tc::smem_u32(bar))
      : "memory");
}

// 32 lanes x 16 consecutive fp32 columns of TMEM into 16 registers per thread.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Fixed-point unit of the epilogue: 2^-50.  Group g (weight 2^(-6(g+2))) enters
// shifted left by 38 - 6g; the last group (g = 7) is rounded by 4 bits.  |sum| <
// 33^2 * 1024 * 2^38 + ... < 2^59 for K <= 1024.
constexpr int kFixBits = 50;
__device__ __forceinline__ long long group_fixed(float v, int g) {
  const long long t = (long long)__float2int_rn(v);   // exact: an integer below 2^24
  const int sh = kFixBits - BETA * (g + 2);
  return sh >= 0 ? (t << sh) : ((t + (1ll << (-sh - 1))) >> -sh);
}

// 32 lanes x 8 consecutive fp32 columns of TMEM at two places.
__device__ __forceinline__ void tmem_ld8x2(uint32_t t0, uint32_t t1, float (&v)[8], float (&w)[8]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(t0), "r"(t1)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = __uint_as_float(r[i]);
    w[i] = __uint_as_float(r[8 + i]);
  }
}

constexpr int kZeroExp = -4000;    // exponent of a row or column of zeros: it never sets the common unit
constexpr int kNanExp = 1 << 20;   // of a column with an infinity or NaN: it always does, and its results are NaN

// a * 2^e as the nearest double (ties to even), integer instructions only, no branch (lanes take every side of one);
// results below the normal range flush to zero, those of a column with kNanExp are NaN.
__device__ __forceinline__ double fixed_to_double(long long a, int e) {
  const unsigned long long sign = (unsigned long long)a & (1ull << 63);
  unsigned long long u = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  const int lz = __clzll((long long)u);
  u <<= lz & 63;                                                     // the leading one at bit 63
  const unsigned long long mant = (u >> 11) + (((u & 0x7FF) + ((u >> 11) & 1)) > 0x400 ? 1 : 0);
  const int ex = 63 - lz + e + 1023;
  // the leading one of mant adds to the exponent field, and so does the carry of a rounding to 2^53
  unsigned long long bits = ((unsigned long long)(unsigned)(ex - 1) << 52) + mant;
  bits = ex >= 0x7FF || bits >= (0x7FFull << 52) ? 0x7FFull << 52 : bits;
  bits = ex <= 0 || a == 0 ? 0ull : bits;
  bits = e >= kNanExp / 2 ? 0x7FF8ull << 48 : bits;
  return __longlong_as_double((long long)(sign | bits));
}

// EPI 0: C = A B.  EPI 1: C += A B.   ea[row], eb[col]: power-of-two exponents of A's rows and B's columns.
template <int EPI>
__global__ void __launch_bounds__(THREADS, 1) gemm_ozaki_kernel(const __grid_constant__ CUtensorMap tmA,
                                                            const __grid_constant__ CUtensorMap tmB,
                                                            const int* __restrict__ ea, const int* __restrict__ eb,
                                                            double* __restrict__ C, int M, long long Ncol, int K,
                                                            int* __restrict__ err, int nd) {
  // nd (1 .. S): leading digits used of each operand (products of weight < nd); the error grows
  // to ~2^(-6 nd) of |A||B|
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // stage s: [nd][BM][BK] bf16 A slices, then [nd][BN][BK] bf16 B slices
  const int ns = stages_for(nd);
  const int stage = nd * (A_SLICE + B_SLICE);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + RING);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* done = empty + MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM;
  const long long n0 = (long long)blockIdx.y * BN;
  const int nkb = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int st = 0; st < ns; ++st) {
      tc::mbar_init(&full[st], 1);
      tc::mbar_init(&empty[st], 1);
    }
    tc::mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(tmem_slot, 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    for (int kb = 0; kb < nkb; ++kb) {
      const int st = kb % ns;
      if (kb >= ns && !tc::mbar_wait(&empty[st], ((kb / ns) + 1) & 1, err)) break;
      uint8_t* sa = smem + st * stage;
      uint8_t* sb = sa + nd * A_SLICE;
      tc::mbar_expect_tx(&full[st], (uint32_t)(nd * (A_SLICE + B_SLICE)));
      for (int p = 0; p < nd; ++p) {
        tma_load_3d(sa + p * A_SLICE, &tmA, kb * BK, m0, p, &full[st]);
        tma_load_3d(sb + p * B_SLICE, &tmB, kb * BK, (int)n0, p, &full[st]);
      }
    }
  } else if (warp == 1 && lane == 0) {
    for (int kb = 0; kb < nkb; ++kb) {
      const int st = kb % ns;
      if (!tc::mbar_wait(&full[st], (kb / ns) & 1, err)) break;
      tc::fence_after();
      const uint8_t* sa = smem + st * stage;
      const uint8_t* sb = sa + nd * A_SLICE;
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
        for (int p = 0; p < nd; ++p)
          for (int q0 = 0; q0 + p < nd; q0 += kSlicesPerMma) {   // weights p+q (0-based) <= nd-1
            const int n = min(kSlicesPerMma, nd - p - q0);
            // slices q0 .. q0+n-1 are consecutive 64-row blocks: their accumulators, groups
            // p+q0 .. p+q0+n-1, are consecutive 64-column blocks of TMEM
            const uint32_t d = tmem + (uint32_t)((p + q0) * BN);
            // every group is first reached with p == 0: the p == 0 products of the first k block
            // and k step initialise the accumulators, every other one accumulates
            const uint32_t acc = (kb > 0 || kk > 0 || p > 0) ? 1u : 0u;
            tc::mma_bf16(d, sdesc_sw64(sa + p * A_SLICE + kk * 32), sdesc_sw64(sb + q0 * B_SLICE + kk * 32),
                         idesc_n(n * BN), acc);
          }
      tc::mma_commit(&empty[st]);
    }
    tc::mma_commit(done);
  }
  __syncwarp();
  const bool ok = tc::mbar_wait(done, 0, err);
  tc::fence_after();
  if (ok && !*(volatile int*)err) {
    // warp w reads TMEM lanes 32 (w % 4) .. +31 (rows) and the 16-column block w / 4
    constexpr int EC = EPI_COLS;
    const int wq = warp & 3, cb = warp >> 2;
    const int row = m0 + wq * 32 + lane;
    const int er = row < M ? ea[row] : 0;
    {
      long long fx[EC];
#pragma unroll
      for (int i = 0; i < EC; ++i) fx[i] = 0;
#pragma unroll 1
      for (int g = 0; g < nd; ++g) {
        float v[EC];
        tmem_ld16(tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(g * BN + cb * EC), v);
#pragma unroll
        for (int i = 0; i < EC; ++i) fx[i] += group_fixed(v[i], g);
      }
      if (row < M) {
        const long long c0 = n0 + cb * EC;
        const int ncb = (int)max(0ll, min((long long)EC, Ncol - c0));
        double* dst = C + c0 * (long long)M + row;
        double old[EC];
        if (EPI == 1) {
#pragma unroll
          for (int i = 0; i < EC; ++i) old[i] = i < ncb ? dst[(long long)i * M] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < EC; ++i) {
          if (i < ncb) {
            const double val = fixed_to_double(fx[i], er + eb[c0 + i] - kFixBits);
            dst[(long long)i * M] = EPI == 1 ? old[i] + val : val;
          }
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// Digits of the columns of a K x Ncol column-major FP64 matrix: for column c with
// max|x| < 2^m, F = round(x 2^(6S-1-m)) (|F| <= 2^(6S-1)) is split into balanced
// base-64 digits t_p (p = 0 most significant), x = 2^e sum_p t_p 2^(-6(p+1)) with
// e = m + 1 written to e_out[c]; t_p goes as bf16 to slices[p][c][k] (K-major).
// Integer arithmetic on the FP64 bit patterns only.
constexpr int kSliceColsPerBlock = 8;   // one warp per column

template <int BITS = BETA>
__device__ __forceinline__ long long round_scaled(long long bits, int m, bool nonzero) {
  const int ex = (int)((bits >> 52) & 0x7FF);
  long long F = 0;   // round(|x| 2^(BITS S-1-m)) <= 2^(BITS S-1)
  if (ex != 0 && nonzero) {
    const unsigned long long mant = ((unsigned long long)bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int rs = m - (ex - 1023 - 52) - (BITS * S - 1);   // >= 54 - BITS S since |x| < 2^m
    if (rs <= 0) F = (long long)(mant << -rs);
    else if (rs < 64) F = (long long)((mant + (1ull << (rs - 1))) >> rs);
  }
  return bits < 0 ? -F : F;
}

// One warp per column, two consecutive k per lane (K is even): 4-byte stores per slice.
__global__ void __launch_bounds__(32 * kSliceColsPerBlock) slice_columns_kernel(const double* __restrict__ X, int K,
                                                                               long long Ncol,
                                                                               __nv_bfloat16* __restrict__ slices,
                                                                               int* __restrict__ e_out,
                                                                               int Kout = 0) {
  // Kout: row length of the slices (>= K, zero-padded; 0: K), for 16-byte TMA rows.
  const int lane = threadIdx.x & 31;
  const long long c = (long long)blockIdx.x * kSliceColsPerBlock + (threadIdx.x >> 5);
  if (c >= Ncol) return;
  const int Ko = Kout > K ? Kout : K;
  const double2* x = reinterpret_cast<const double2*>(X + c * (long long)K);
  const int K2 = K / 2;
  unsigned long long mx = 0;
  for (int k = lane; k < K2; k += 32) {
    const double2 v = x[k];
    const unsigned long long a = (unsigned long long)__double_as_longlong(v.x) & 0x7FFFFFFFFFFFFFFFull;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v.y) & 0x7FFFFFFFFFFFFFFFull;
    mx = a > mx ? a : mx;
    mx = b > mx ? b : mx;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = t > mx ? t : mx;
  }
  const int emax = (int)((mx >> 52) & 0x7FF);
  const int m = mx == 0 ? 0 : emax - 1023 + 1;   // max|x| < 2^m
  if (lane == 0) e_out[c] = m + 1;
  const long long slice_stride = Ncol * (long long)Ko;
  __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(slices + c * (long long)Ko);
  for (int k = K2 + lane; k < Ko / 2; k += 32)
#pragma unroll
    for (int p = 0; p < S; ++p) out[p * (slice_stride / 2) + k] = __floats2bfloat162_rn(0.f, 0.f);
  for (int k = lane; k < K2; k += 32) {
    const double2 v = x[k];
    long long F0 = round_scaled(__double_as_longlong(v.x), m, mx != 0);
    long long F1 = round_scaled(__double_as_longlong(v.y), m, mx != 0);
#pragma unroll
    for (int p = S - 1; p > 0; --p) {
      const int d0 = (int)(((F0 + 32) & 63) - 32), d1 = (int)(((F1 + 32) & 63) - 32);
      out[p * (slice_stride / 2) + k] = __floats2bfloat162_rn((float)d0, (float)d1);
      F0 = (F0 - d0) >> BETA;
      F1 = (F1 - d1) >> BETA;
    }
    out[k] = __floats2bfloat162_rn((float)F0, (float)F1);
  }
}

// ---------------------------------------------------------------------------------------------
// The plane-wave transforms of the 1D operator with the same digits.  Phi(m, p) = c + i d is symmetric under k -> -k and
// xi -> -xi, so with E = x_p + x_p' and O = x_p - x_p' of the mirror pairs (p, p')
//   A = sum_p c E, B = sum_p d O,   X^(m) = A + i B, X^(m') = A - i B
// (the adjoint i Phi^H: A - i B and A + i B), two real matrices of half the rows and columns instead of
// the 2 x 2 real embedding of a complex one: a quarter of the digit products, an eighth of the table.
//   B operand: real columns 2 c + (0 re, 1 im) of node c, plane 0 = E, plane 1 = O: rows plane 2 ncols + 2 c + o
//   A operand: rows plane hm + m, hm = M / 2 (plane 0 = c, plane 1 = d)
// One CTA computes A, drains TMEM to FP64 registers, computes B into the same accumulators (its first loads are in
// flight meanwhile), and writes both members of every output pair.  All 16 warps drain, warp 0 loads and warp 1 issues
// between (two warps more had left 96 registers a thread and spilled the drain).
//   MODE 0: Y = Phi X.   MODE 1: Y = i Phi^H X.
// The table's digits dominated the L2 traffic of the embedded product (1 MB per 64 nodes, a quarter of it per CTA;
// now 0.5 MB per 32 nodes for both planes).  Half the columns also leave room for 7 bits a digit: |t| <= 64, and 8
// products of K <= 256 pairs stay at 8 * 64^2 * 256 = 2^23, exact in FP32.  Eight digits carry 56 bits of a column's
// largest entry, more than FP64 keeps of a sum of K such terms; seven (28 products of digits instead of 36) carry 49, one more
// than eight of 6 bits.  With slicing, per transform: 333 -> 184 us (16 problems of 960 nodes,
// 256 x 256), 240 -> 119 us (4 of 720 nodes, 512 x 512: 180 CTAs on 152 SMs); with eight digits of 6 bits, FP64 additions in the
// epilogue and all of it inlined 219 and 158 us.  A CTA of 256 x 256 takes 36 us: 2 until its first stage, 8 of MMAs a
// plane, 2 to read plane 0, the rest the conversions and stores of the results.
// ---------------------------------------------------------------------------------------------
constexpr int PAIR_BITS = 7, PAIR_MAX_K = 256;   // bits per digit, pairs per row
constexpr int kPairFixBits = 55;                 // unit 2^-55; |sum| <= K / 4 = 2^6, |A +- B| <= 2^7 of it
// Two neighbouring groups are one 32-bit integer (2^23 2^7 + 2^23); pair j (groups 2j, 2j + 1) has weight 2^(-21 - 14 j),
// the last one is rounded by 8 bits.
__device__ __forceinline__ long long pair_fixed(const int (&c)[4]) {
  return ((long long)c[0] << 34) + ((long long)c[1] << 20) + ((long long)c[2] << 6) + ((c[3] + 128) >> 8);
}
// The integer value of a group: up to 2^22 (K <= 128) by the rounding of an addition, which is two instructions of
// the FP32 pipe; the conversion instruction runs at an eighth of their rate.
template <bool SMALL>
__device__ __forceinline__ int group_int(float v) {
  if constexpr (SMALL) return __float_as_int(__fadd_rn(v, 12582912.f)) - 0x4B400000;   // 1.5 2^23
  else return __float2int_rn(v);
}
// a and b of units 2^ea and 2^eb in the larger of the two, which ea becomes
__device__ __forceinline__ void pair_align(long long& a, int& ea, long long& b, int eb) {
  const int d = eb - ea, sa = min(max(d, 0), 62), sb = min(max(-d, 0), 62);
  a = (a + ((1ll << sa) >> 1)) >> sa;
  b = (b + ((1ll << sb) >> 1)) >> sb;
  ea = max(ea, eb);
}

// The pair of results of one node from A and B (units 2^(ea + xa), 2^(eb + xb)), as integers of a common unit with one
// conversion per result: the FP64 additions of the pairs cost 64 cycles of an SM quarter each.  Not inlined: eight copies
// of it are read from the instruction cache once per CTA (20,000 of its 75,000 cycles, 37,000 when it is cold).
template <int MODE>
__device__ __noinline__ void pair_store(long long ar, long long ai, long long br, long long bi, int ea, int eb, int2 xa,
                                        int2 xb, double2* p, double2* q) {
  int e0 = ea + xa.x, e1 = ea + xa.y;
  pair_align(ar, e0, bi, eb + xb.y);   // the results of Re A and Im B
  pair_align(ai, e1, br, eb + xb.x);   // and of Im A and Re B
  if (MODE == 0) {
    *p = make_double2(fixed_to_double(ar - bi, e0), fixed_to_double(ai + br, e1));
    *q = make_double2(fixed_to_double(ar + bi, e0), fixed_to_double(ai - br, e1));
  } else {
    *p = make_double2(fixed_to_double(br - ai, e1), fixed_to_double(ar + bi, e0));
    *q = make_double2(fixed_to_double(-(ai + br), e1), fixed_to_double(ar - bi, e0));
  }
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1) gemm_pairs_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const int* __restrict__ ea,
    const int* __restrict__ eb, double2* __restrict__ Y, int M, long long Ncol2, int K, int* __restrict__ err,
    const int* __restrict__ mask, int cols_per_problem, int nd, const int* __restrict__ nd_pp) {
  // Ncol2, cols_per_problem: real columns (two per node).  nd (1 .. S): leading digits used of each operand; nd_pp
  // (optional): digits per problem, the tile takes the largest of its problems.  A column tile whose
  // problems are all inactive has nothing to compute.  Grid: all tiles in x, row tiles first (columns in y end at 65,535
  // tiles, two million nodes).
  const int hm = M / 2, row_tiles = (hm + BM - 1) / BM, m0 = (int)(blockIdx.x % row_tiles) * BM;
  const long long n0 = (long long)(blockIdx.x / row_tiles) * BN;
  if (mask || nd_pp) {
    const long long c0 = n0, c1 = min(Ncol2, c0 + BN) - 1;
    bool any = false;
    int ndt = 1;
    for (long long b = c0 / cols_per_problem; b <= c1 / cols_per_problem; ++b) {
      const bool on = !mask || mask[b] != 0;
      any |= on;
      if (nd_pp && on) ndt = max(ndt, min(S, max(1, nd_pp[b])));
    }
    if (!any) return;
    if (nd_pp) nd = ndt;
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ns = stages_for(nd);
  const int stage = nd * (A_SLICE + B_SLICE);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + RING);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* done = empty + MAX_STAGES;   // [2] the accumulators of a plane are complete
  uint64_t* drained = done + 2;          // plane 0 has been read out of TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int st = 0; st < ns; ++st) {
      tc::mbar_init(&full[st], 1);
      tc::mbar_init(&empty[st], 1);
    }
    tc::mbar_init(&done[0], 1);
    tc::mbar_init(&done[1], 1);
    tc::mbar_init(drained, THREADS / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(tmem_slot, 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  auto load = [&](int it0, int it1) {
    for (int it = it0; it < it1; ++it) {
      const int st = it % ns, ph = it / nkb, kb = it - ph * nkb;
      if (it >= ns && !tc::mbar_wait(&empty[st], ((it / ns) + 1) & 1, err)) break;
      uint8_t* sa = smem + st * stage;
      uint8_t* sb = sa + nd * A_SLICE;
      tc::mbar_expect_tx(&full[st], (uint32_t)(nd * (A_SLICE + B_SLICE)));
      for (int p = 0; p < nd; ++p) {
        tma_load_3d(sa + p * A_SLICE, &tmA, kb * BK, ph * hm + m0, p, &full[st]);
        tma_load_3d(sb + p * B_SLICE, &tmB, kb * BK, (int)(ph * Ncol2 + n0), p, &full[st]);
      }
    }
  };
  auto multiply = [&](int ph) {
    for (int kb = 0; kb < nkb; ++kb) {
      const int it = ph * nkb + kb, st = it % ns;
      if (!tc::mbar_wait(&full[st], (it / ns) & 1, err)) return;
      tc::fence_after();
      const uint8_t* sa = smem + st * stage;
      const uint8_t* sb = sa + nd * A_SLICE;
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
        for (int p = 0; p < nd; ++p)
          for (int q0 = 0; q0 + p < nd; q0 += kSlicesPerMma) {   // as in gemm_ozaki_kernel
            const int n = min(kSlicesPerMma, nd - p - q0);
            tc::mma_bf16(tmem + (uint32_t)((p + q0) * BN), sdesc_sw64(sa + p * A_SLICE + kk * 32),
                         sdesc_sw64(sb + q0 * B_SLICE + kk * 32), idesc_n(n * BN),
                         (kb > 0 || kk > 0 || p > 0) ? 1u : 0u);
          }
      tc::mma_commit(&empty[st]);
    }
    tc::mma_commit(&done[ph]);
  };
  {
    // warp w reads TMEM lanes 32 (w % 4) .. +31 (rows) and the 16 real columns (8 nodes) of block w / 4, eight at a time
    // (16 left no registers for plane 0's results)
    constexpr int EC = EPI_COLS;
    const int wq = warp & 3, cb = warp >> 2;
    const int row = m0 + wq * 32 + lane;
    const long long c0 = n0 + cb * EC;
    const int ncb = (int)max(0ll, min((long long)EC, Ncol2 - c0));
    const bool in = row < hm;
    const uint32_t tbase = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(cb * EC);
    const bool small = K <= PAIR_MAX_K / 2;
    auto drain = [&](int half, long long* out) {
      int c[8][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v[8], w[8];
        const uint32_t t = tbase + (uint32_t)(2 * j * BN + 8 * half);
        const bool two = 2 * j + 1 < nd;
        if (2 * j < nd) tmem_ld8x2(t, two ? t + BN : t, v, w);
        if (small) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            c[i][j] = 2 * j < nd ? group_int<true>(v[i]) * 128 + (two ? group_int<true>(w[i]) : 0) : 0;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            c[i][j] = 2 * j < nd ? group_int<false>(v[i]) * 128 + (two ? group_int<false>(w[i]) : 0) : 0;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = pair_fixed(c[i]);
    };
    // plane 0, and as many loads of plane 1 as the ring takes before the accumulators are read
    const int ahead = min(nkb + ns, 2 * nkb);
    if (warp == 0 && lane == 0) load(0, ahead);
    if (warp == 1 && lane == 0) multiply(0);
    __syncwarp();
    long long va[EC];
    bool ok = tc::mbar_wait(&done[0], 0, err);
    tc::fence_after();
    if (ok) {
      drain(0, va);
      drain(1, va + 8);
    }
    tc::fence_before();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(drained);
    if (warp == 0 && lane == 0) load(ahead, 2 * nkb);
    if (warp == 1 && lane == 0 && tc::mbar_wait(drained, 0, err)) {
      tc::fence_after();
      multiply(1);
    }
    __syncwarp();
    const int ea0 = in ? ea[row] - kPairFixBits : 0, ea1 = in ? ea[hm + row] - kPairFixBits : 0;
    if (ok) ok = tc::mbar_wait(&done[1], 0, err);
    tc::fence_after();
    if (ok && !*(volatile int*)err) {
      double2* y = Y + c0 / 2 * M;
      const int mr = M - 1 - row;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        long long vb[8];
        drain(half, vb);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = 8 * half + 2 * i;
          if (!in || col >= ncb) continue;
          const int2 xa = make_int2(eb[c0 + col], eb[c0 + col + 1]);
          const int2 xb = make_int2(eb[Ncol2 + c0 + col], eb[Ncol2 + c0 + col + 1]);
          double2* yn = y + (long long)(4 * half + i) * M;
          pair_store<MODE>(va[col], va[col + 1], vb[2 * i], vb[2 * i + 1], ea0, ea1, xa, xb, yn + row, yn + mr);
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// Digits of E and O of every node's complex column (K entries, K even and at most 512), one warp per real column (E re,
// E im, O re, O im of a node: four warps share its loads through the L1; one warp per node left a chain of 1,900
// instructions, 14 us at 1,920 nodes of 256 entries against 11; bound by the FP64 additions, the pipe is 76% busy), two
// consecutive pairs per lane and pass; the column
// stays in registers between its maximum and its digits.  Rows of Kout entries (>= K / 2, zero-padded).  nd, nd_pp:
// the digits gemm_pairs_kernel reads for the node's tile.  PASSES of 64 entries cover Kout (1, 2 or 4).
constexpr int kSlicePairNodes = 2;   // per block of eight warps
template <int PASSES>
__global__ void __launch_bounds__(128 * kSlicePairNodes) slice_pairs_kernel(
    const double2* __restrict__ X, int K, long long ncols, __nv_bfloat16* __restrict__ slices, int* __restrict__ e_out,
    const int* __restrict__ mask, int nodes_per_problem, int Kout, int nd, const int* __restrict__ nd_pp) {
  const int lane = threadIdx.x & 31, o = (threadIdx.x >> 5) & 3;
  const long long c = (long long)blockIdx.x * kSlicePairNodes + (threadIdx.x >> 7);
  if (c >= ncols || (mask && !mask[c / nodes_per_problem])) return;
  int ndt = nd < 1 ? 1 : (nd > S ? S : nd);
  if (nd_pp) {
    constexpr int NT = BN / 2;
    const long long c0 = c / NT * NT, c1 = min(ncols, c0 + NT) - 1;
    ndt = 1;
    for (long long b = c0 / nodes_per_problem; b <= c1 / nodes_per_problem; ++b)
      if (!mask || mask[b] != 0) ndt = max(ndt, min(S, max(1, nd_pp[b])));
  }
  const int h = K / 2;
  const double* x = reinterpret_cast<const double*>(X + c * K) + (o & 1);
  const bool odd = o >> 1;
  long long v[PASSES][2];
  unsigned long long mx = 0;
#pragma unroll
  for (int t = 0; t < PASSES; ++t)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int p = 64 * t + 2 * lane + u;
      double w = 0.0;
      if (p < h) {
        const double a = x[2 * p], b = x[2 * (K - 1 - p)];
        w = odd ? a - b : a + b;
      }
      v[t][u] = __double_as_longlong(w);
      const unsigned long long m = (unsigned long long)v[t][u] & 0x7FFFFFFFFFFFFFFFull;
      mx = m > mx ? m : mx;
    }
  for (int q = 16; q > 0; q >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, mx, q);
    mx = t > mx ? t : mx;
  }
  const int m = mx == 0 ? 0 : (int)((mx >> 52) & 0x7FF) - 1023 + 1;   // max|x| < 2^m
  const bool finite = mx < 0x7FFull << 52, digits = mx != 0 && finite;
  const long long Ncol2 = 2 * ncols, slice_stride = 2 * Ncol2 * (long long)Kout;
  const long long r = (o >> 1) * Ncol2 + 2 * c + (o & 1);
  if (lane == 0) e_out[r] = mx == 0 ? kZeroExp : finite ? m + 1 : kNanExp;
  __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(slices + r * Kout);
#pragma unroll
  for (int t = 0; t < PASSES; ++t) {
    const int k = 32 * t + lane;
    if (2 * k >= Kout) continue;
    long long F0 = round_scaled<PAIR_BITS>(v[t][0], m, digits);
    long long F1 = round_scaled<PAIR_BITS>(v[t][1], m, digits);
#pragma unroll
    for (int p = S - 1; p > 0; --p) {
      const int d0 = (int)(((F0 + 64) & 127) - 64), d1 = (int)(((F1 + 64) & 127) - 64);
      if (p < ndt) out[p * (slice_stride / 2) + k] = __floats2bfloat162_rn((float)d0, (float)d1);
      F0 = (F0 - d0) >> PAIR_BITS;
      F1 = (F1 - d1) >> PAIR_BITS;
    }
    out[k] = __floats2bfloat162_rn((float)F0, (float)F1);
  }
}

}  // namespace oz
}  // namespace wg
