// Transverse subband eigensolve (mode space) on the device (sm_103a).
//
// For every valley v and x slice the reference builds the Ny x Ny finite-difference
// Hamiltonian of the confinement direction (eval_transversal_Hamiltonian.m:20-37) and asks
// eigs for the n_of_modes eigenpairs of smallest magnitude (solve_bandstructure.m:17-33),
// then fixes the signs of valley 1 against its first slice (solve_subbands.m:22-40).
//
// Ht is tridiagonal and symmetric except for its copied end rows; with positive
// off-diagonal products T = D^-1 Ht D is symmetric tridiagonal for a diagonal D
// (d_{i+1} / d_i = sqrt(Ht(i+1,i) / Ht(i,i+1))), with the same eigenvalues and the
// eigenvectors v = D w.  Per slice:
//   subband_coarse_kernel   one warp per slice (problem, valley, x), all in FP32: Sturm counts (signs of the LDL^T
//     pivots of T - x) around 0, then multisection of the eigenvalues with index in [n0 - nm, n0 + nm),
//     n0 = #(< 0), to 1e-6 of the spectral radius (the candidates share the 32 lanes, g lanes count at g interior
//     points of a candidate's interval per step); the nm of smallest magnitude are a contiguous run around zero.
//   subband_refine_kernel   one lane per (slice, mode), FP64: Rayleigh quotient steps of the twisted factorisation
//     of T - lambda (Dhillon and Parlett, "Orthogonal eigenvectors and relative gaps", SIAM J. Matrix Anal.
//     Appl. 25 (2004) 858-899): top-down pivots D+, bottom-up pivots D-, the twist index r of smallest |gamma_r|,
//     z_r = 1 and the one-term recurrences out of r; lambda += gamma_r / |z|^2 squares the error over the gap, so from
//     1e-6 two steps reach rounding level and the third factorisation gives the vector.  The negative pivots
//     count the eigenvalues below lambda: it is eigenvalue k, or the slice goes to
//   subband_bisect_kernel   one warp per listed slice: FP64 multisection to the end and the vectors from it.  It
//     takes what the others cannot vouch for: two eigenvalues closer than the FP32 bracket, a tie of |lambda| at the
//     edge of the run, entries outside the FP32 range, invalid data (which it reports).
//   subband_cleanup_kernel  one warp per (problem, x >= 1, mode) of valley 1: v -> -v when
//                           its overlap with the same mode of slice 1 is below -1/2.
// A handle solves a batch of independent problems (gate or bias points) in one launch.
// v = D w normalised in the 2-norm and signed by its last entry (solve_bandstructure.m:28-30).
//
// Bound by the FP64 pipe (a warp instruction takes a quarter's pipe for 64 cycles however many lanes are on):
// the multisection needed ~20 FP64 sweeps with a division per row for each slice's own warp, the refinement takes
// three factorisations with a 4-operation reciprocal for 32 modes (several slices) at once.
// 25,664 slices of 71 rows, 8 modes: 34.0 -> 2.1 ms; one gate point of 234 slices, 67 rows, 4 modes (host call):
// 0.93 -> 0.39 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>

#include "recip.cuh"
#include "wigner_gb300.h"

using wg::fast_rcp;

namespace {

constexpr int kMaxModes = 32;
constexpr int kMaxNy = 1024;

struct SliceShared {
  double *a, *b, *b2, *rr, *lam;
  float *af, *b2f;   // FP32 copies of a and b^2 for the coarse bisection
};

// per warp: a, b, b2, rr [ny] doubles, lam [2 kMaxModes] doubles, af, b2f [ny] floats
__host__ __device__ constexpr int slice_doubles(int ny) { return 5 * ny + 2 * kMaxModes; }

__device__ __forceinline__ SliceShared slice_shared(double* base, int ny) {
  SliceShared s;
  s.a = base;
  s.b = base + ny;
  s.b2 = base + 2 * ny;
  s.rr = base + 3 * ny;
  s.lam = base + 4 * ny;
  s.af = reinterpret_cast<float*>(base + 4 * ny + 2 * kMaxModes);
  s.b2f = s.af + ny;
  return s;
}

__device__ __forceinline__ double guard(double q, double pivmin) { return fabs(q) < pivmin ? -pivmin : q; }

// Number of eigenvalues of T below x: negative pivots of T - x = L D L^T.
__device__ int sturm_count(const SliceShared& s, int n, double x, double pivmin) {
  double q = guard(s.a[0] - x, pivmin);
  int c = q < 0.0;
  for (int i = 1; i < n; ++i) {
    q = guard(s.a[i] - x - s.b2[i - 1] / q, pivmin);
    c += q < 0.0;
  }
  return c;
}

// The same count in FP32 (coarse: wrong only within ~ny FP32 ulps of an eigenvalue).
__device__ int sturm_count32(const SliceShared& s, int n, float x, float pivmin) {
  float q = s.af[0] - x;
  q = fabsf(q) < pivmin ? -pivmin : q;
  int c = q < 0.f;
  for (int i = 1; i < n; ++i) {
    q = s.af[i] - x - s.b2f[i - 1] / q;
    q = fabsf(q) < pivmin ? -pivmin : q;
    c += q < 0.f;
  }
  return c;
}

__device__ __forceinline__ double hop(double t0, double ma, double mb) { return -2.0 * t0 / (ma + mb); }

// Slices left to the bisection: list[0 .. *count), each once (flag per slice).
struct FallbackList {
  int *count, *flag, *list;
  __device__ void add(int slice) const {
    if (atomicExch(&flag[slice], 1) == 0) list[atomicAdd(count, 1)] = slice;
  }
};

// The count in FP32 with fast divisions: exact for a matrix a few FP32 ulps of the spectral radius away.
__device__ __forceinline__ int coarse_count(const float* a, const float* b2, int n, float x, float pivmin) {
  float q = a[0] - x;
  q = fabsf(q) < pivmin ? -pivmin : q;
  int c = q < 0.f;
#pragma unroll 4
  for (int i = 1; i < n; ++i) {
    q = a[i] - x - __fdividef(b2[i - 1], q);
    q = fabsf(q) < pivmin ? -pivmin : q;
    c += q < 0.f;
  }
  return c;
}

__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// Of eigenvalue kp > 0 and eigenvalue kn < 0 of T, whose magnitudes lie in (lo, hi): is |lambda_kn| the smaller?  FP64
// counts at 16 magnitudes of either sign by the lanes of a warp, four rounds (the interval shrinks 17-fold in each); -1: not
// settled.  a, b2: the slice's T in global memory.  A slice left to the bisection costs a chain of 500 us however
// few there are; one round costs 15 us.
__device__ int tie_smaller(const double* a, const double* b2, int n, int kp, int kn, double lo, double hi,
                           double pivmin) {
  const int lane = threadIdx.x & 31;
  const unsigned long long pivbits = abs_bits(pivmin);
  for (int round = 0; round < 4; ++round) {
    const double step = (hi - lo) * (1.0 / 17.0), s = lo + ((lane >> 1) + 1) * step, x = lane & 1 ? -s : s;
    double q = a[0] - x;
    if (abs_bits(q) < pivbits) q = -pivmin;
    int c = q < 0.0;
    for (int i = 1; i < n; ++i) {
      q = fma(-b2[i - 1], fast_rcp(q), a[i] - x);
      if (abs_bits(q) < pivbits) q = -pivmin;
      c += q < 0.0;
    }
    // inside: the eigenvalue's magnitude is below s
    const unsigned in = __ballot_sync(0xffffffffu, lane & 1 ? c <= kn : c > kp);
    const unsigned pos = in & 0x55555555u, neg = (in >> 1) & 0x55555555u;
    const int fp = pos ? (__ffs(pos) - 1) / 2 : 16, fn = neg ? (__ffs(neg) - 1) / 2 : 16;
    if (fp != fn) return fn < fp;
    const double l = lo + fp * step;
    hi = fp == 16 ? hi : l + step;
    lo = l;
  }
  return -1;
}

// Shared memory of the coarse stage per warp: a, b^2 [ny] and up to 2 nm + 1 candidates.
__host__ __device__ constexpr int coarse_floats(int ny) { return 2 * ny + 2 * kMaxModes + 2; }

// Width of the FP32 brackets, and what two of them may be apart and still be confused, in units of the radius.
constexpr float kCoarseTol = 1e-6f, kCoarseMargin = 2e-5f;

// E[slice][k] <- the FP32 estimate of eigenvalue kfirst[slice] + k (kfirst = -1: left to the bisection).
__global__ void __launch_bounds__(128) subband_coarse_kernel(const double* __restrict__ me_y,
                                                             const double* __restrict__ pot, float t0, int nslice,
                                                             int nv, int nx, int ny, int nm, double* __restrict__ E,
                                                             int* __restrict__ kfirst, double t0d, double* dplus,
                                                             double* dminus, FallbackList fb) {
  // dplus, dminus: the refinement's scratch, here T of a slice with a tie
  extern __shared__ float smf[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slice = blockIdx.x * (blockDim.x >> 5) + warp;   // slice = (problem * nv + v) * nx + x
  if (slice >= nslice) return;
  float* a = smf + (size_t)warp * coarse_floats(ny);
  float* b2 = a + ny;
  float* lam = b2 + ny;   // up to 2 nm + 1 candidates
  const double* m = me_y + (size_t)slice * ny;
  const double* V = pot + ((size_t)(slice / (nv * nx)) * nx + slice % nx) * ny;
  auto hopf = [&](int i) { return -2.f * t0 / ((float)m[i] + (float)m[i + 1]); };   // rows i, i + 1
  bool bad = false;
  float glo = INFINITY, ghi = -INFINITY, bmax = 0.f;
  for (int i = lane; i < ny; i += 32) {
    const int r = i == 0 ? 1 : (i == ny - 1 ? ny - 2 : i);
    const float lo = hopf(r - 1), up = hopf(r);
    a[i] = -(lo + up) + (float)V[r];
    // Ht(i, i+1) Ht(i+1, i); rows 0 and ny - 1 copy rows 1 and ny - 2
    const float p = i == ny - 1 ? 0.f : (i == 0 ? up : hopf(i)) * (i + 1 == ny - 1 ? hopf(ny - 3) : hopf(i));
    b2[i] = p;
    bad = bad || !isfinite(a[i]) || !isfinite(p) || (i < ny - 1 && !(p > 0.f));
    bmax = fmaxf(bmax, p);
  }
  __syncwarp();
  for (int i = lane; i < ny; i += 32) {
    const float rad = sqrtf(b2[i]) + (i > 0 ? sqrtf(b2[i - 1]) : 0.f);
    glo = fminf(glo, a[i] - rad);
    ghi = fmaxf(ghi, a[i] + rad);
  }
  for (int o = 16; o; o >>= 1) {
    glo = fminf(glo, __shfl_xor_sync(0xffffffffu, glo, o));
    ghi = fmaxf(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
  }
  const float gnorm = fmaxf(fabsf(glo), fabsf(ghi)), pivmin = FLT_MIN * fmaxf(1.f, bmax);
  bad = __any_sync(0xffffffffu, bad || !(gnorm < 1e30f));
  int first = -1;
  if (!bad) {
    glo -= 1e-5f * gnorm;
    ghi += 1e-5f * gnorm;
    // the counts a little below and above 0 bound n0 from both sides
    const float zero = 4e-6f * gnorm;
    const int cz = lane < 2 ? coarse_count(a, b2, ny, lane == 0 ? -zero : zero, pivmin) : 0;
    const int na = __shfl_sync(0xffffffffu, cz, 0), nb = __shfl_sync(0xffffffffu, cz, 1);
    const int c0 = max(0, na - nm), c1 = min(ny, nb + nm), nc = c1 - c0;
    // more candidates than the window holds (a potential far above the other levels leaves all of them within the
    // band around 0): nothing is located, the slice goes to the bisection
    bad = nb - na != 0 && nb - na != 1;
    for (int cb = 0; cb < nc && !bad; cb += 32) {
      const int n = min(32, nc - cb), g = 32 / n, c = lane / g, j = lane % g;
      const bool mine = c < n;
      const int k = c0 + cb + (mine ? c : 0);
      const unsigned gmask = (g == 32 ? 0xffffffffu : ((1u << g) - 1u)) << (mine ? c * g : 0);
      float lo = glo, hi = ghi;
      for (int it = 0; it < 64; ++it) {
        const bool open = mine && hi - lo > kCoarseTol * gnorm;
        if (!__any_sync(0xffffffffu, open)) break;
        const float step = (hi - lo) / (g + 1), p = lo + (j + 1) * step;
        const bool above = open && (p >= hi || (p > lo && coarse_count(a, b2, ny, p, pivmin) > k));
        const unsigned vote = __ballot_sync(0xffffffffu, above) & gmask;
        if (open) {
          const int jf = vote ? __ffs(vote) - 1 - c * g : g;
          const float nlo = jf == 0 ? lo : fmaxf(lo, lo + jf * step);
          const float nhi = jf == g ? hi : fminf(hi, lo + (jf + 1) * step);
          lo = nlo;
          hi = nhi;
        }
      }
      if (mine && j == 0) lam[cb + c] = 0.5f * (lo + hi);
    }
    __syncwarp();
    if (!bad) {
      // the nm of smallest magnitude: grow a window outwards from the sign change
      int lo = -1, hi = 0;
      while (hi < nc && lam[hi] < 0.f) ++hi;
      lo = hi - 1;
      for (int t = 0; t < nm; ++t) {
        if (hi < nc && (lo < 0 || fabsf(lam[hi]) <= fabsf(lam[lo]))) ++hi;
        else --lo;
      }
      // the last one taken and the first one left out on the other side: a tie in FP32 is settled by FP64 counts
      const float margin = 2 * kCoarseMargin * gnorm;
      const bool low = lo >= 0 && hi - 1 > lo && lam[hi - 1] > 0.f && fabsf(lam[lo]) - lam[hi - 1] < margin;
      const bool high = hi < nc && lo + 1 < hi && lam[lo + 1] < 0.f && fabsf(lam[hi]) - fabsf(lam[lo + 1]) < margin;
      bad = low && high;
      if (low != high) {
        const int p = low ? hi - 1 : hi, n = low ? lo : lo + 1;   // the positive and the negative candidate
        double* ta = dplus + (size_t)slice * ny * nm;
        double* tb = dminus + (size_t)slice * ny * nm;
        for (int i = lane; i < ny; i += 32) {
          const int r = i == 0 ? 1 : (i == ny - 1 ? ny - 2 : i);
          ta[i] = -(hop(t0d, m[r - 1], m[r]) + hop(t0d, m[r], m[r + 1])) + V[r];
          tb[i] = i == ny - 1 ? 0.0
                              : (i == 0 ? hop(t0d, m[1], m[2]) : hop(t0d, m[i], m[i + 1])) *
                                    (i + 1 == ny - 1 ? hop(t0d, m[ny - 3], m[ny - 2]) : hop(t0d, m[i], m[i + 1]));
        }
        __syncwarp();
        const float x = fminf(lam[p], -lam[n]), y = fmaxf(lam[p], -lam[n]);
        const int neg = tie_smaller(ta, tb, ny, c0 + p, c0 + n, (double)fmaxf(x - margin, 0.f), (double)(y + margin),
                                    1e-30 * (double)gnorm);
        bad = neg < 0;
        const int shift = low ? (neg == 1 ? -1 : 0) : (neg == 0 ? 1 : 0);
        lo += shift;
        hi += shift;
        // the window moved past another candidate that close: left to the bisection
        if (shift < 0 && lo >= 0 && hi - 1 > lo && lam[hi - 1] > 0.f && fabsf(lam[lo]) - lam[hi - 1] < margin) bad = true;
        if (shift > 0 && hi < nc && lo + 1 < hi && lam[lo + 1] < 0.f && fabsf(lam[hi]) - fabsf(lam[lo + 1]) < margin)
          bad = true;
      }
      first = c0 + lo + 1;
      for (int k = lane; k < nm; k += 32) E[(size_t)slice * nm + k] = lam[lo + 1 + k];
    }
  }
  if (lane == 0) {
    kfirst[slice] = bad ? -1 : first;
    if (bad) fb.add(slice);
  }
}

// Shared memory of the refinement: per slice a, b^2, b [ny], and the slices a block of one warp takes (32 / nm
// where their data fit in 40 KB).
__host__ __device__ constexpr int refine_doubles(int ny) { return 3 * ny; }
int refine_slices(int ny, int nm) {
  return std::max(1, std::min(32 / nm, (int)(40 * 1024 / (sizeof(double) * refine_doubles(ny)))));
}

__global__ void __launch_bounds__(32) subband_refine_kernel(const double* __restrict__ me_y,
                                                            const double* __restrict__ pot, double t0, int nslice,
                                                            int nv, int nx, int ny, int nm, int sl,
                                                            double* __restrict__ E, double* __restrict__ Vsub,
                                                            double* __restrict__ dplus, double* __restrict__ dminus,
                                                            const int* __restrict__ kfirst, FallbackList fb) {
  extern __shared__ double smem[];
  __shared__ double r0s[32], r1s[32], gns[32];
  const int lane = threadIdx.x, s0 = blockIdx.x * sl;
  // T of every slice of the block; rows 0 and ny - 1 of Ht copy rows 1 and ny - 2
  for (int q = 0; q < sl && s0 + q < nslice; ++q) {
    const int slice = s0 + q;
    double* a = smem + (size_t)q * refine_doubles(ny);
    double *b2 = a + ny, *b = b2 + ny;
    const double* m = me_y + (size_t)slice * ny;
    const double* V = pot + ((size_t)(slice / (nv * nx)) * nx + slice % nx) * ny;
    for (int i = lane; i < ny; i += 32) b[i] = i < ny - 1 ? hop(t0, m[i], m[i + 1]) : 0.0;
    __syncwarp();
    const double u0 = b[1], l0 = b[0], u1 = b[ny - 2], l1 = b[ny - 3];
    float g = 0.f;
    for (int i = lane; i < ny; i += 32) {
      const int r = i == 0 ? 1 : (i == ny - 1 ? ny - 2 : i);
      const double h = b[i];
      a[i] = -(b[r - 1] + b[r]) + V[r];
      b2[i] = i == 0 ? u0 * l0 : i == ny - 2 ? u1 * l1 : h * h;
      g = fmaxf(g, fabsf((float)a[i]) + 2.f * fmaxf(fabsf((float)b[r - 1]), fabsf((float)b[r])));
    }
    __syncwarp();
    if (lane == 0) {
      b[0] = -sqrt(u0 * l0);
      r0s[q] = sqrt(u0 / l0);          // v_0 = w_0 / (d_1 / d_0) in units of the interior's d
    }
    if (lane == 1) {
      b[ny - 2] = -sqrt(u1 * l1);
      r1s[q] = sqrt(l1 / u1);
    }
    for (int o = 16; o; o >>= 1) g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, o));
    if (lane == 0) gns[q] = g;
    __syncwarp();
  }
  const int q = lane / nm, k = lane % nm, slice = s0 + q;
  if (q >= sl || slice >= nslice) return;
  const int kf = kfirst[slice];
  if (kf < 0) return;
  const double* a = smem + (size_t)q * refine_doubles(ny);
  const double *b2 = a + ny, *b = b2 + ny;
  // pivots below 1e-30 of the radius (some are exactly zero at a converged lambda) are moved to -1e-30 of it: far
  // below their rounding, and their reciprocals and the next pivots stay in range
  const double gnorm = gns[q], pivmin = 1e-30 * gnorm, atol = 4.0 * DBL_EPSILON * gnorm;
  const unsigned long long pivbits = abs_bits(pivmin);
  const double lam0 = E[(size_t)slice * nm + k];
  double* dp = dplus + (size_t)slice * ny * nm + k;    // 1 / D+, then the vector [i][mode]
  double* dm = dminus + (size_t)slice * ny * nm + k;   // 1 / D-
  double lam = lam0, z0 = 0.0, z1 = 0.0, nint = 0.0;
  bool ok = false, sure = false;
  for (int it = 0; it < 8; ++it) {
    double qp = a[0] - lam;
    if (abs_bits(qp) < pivbits) qp = -pivmin;
    int neg = qp < 0.0;
    double ri = fast_rcp(qp);
    dp[0] = ri;
#pragma unroll 4
    for (int i = 1; i < ny; ++i) {
      qp = fma(-b2[i - 1], ri, a[i] - lam);
      if (abs_bits(qp) < pivbits) qp = -pivmin;
      neg += (int)((unsigned long long)__double_as_longlong(qp) >> 63);
      ri = fast_rcp(qp);
      dp[(size_t)i * nm] = ri;
    }
    // gamma_i = D+_i + D-_i - (a_i - lambda) = D-_i - b2_{i-1} / D+_{i-1}
    int r = ny - 1;
    double gam = qp;
    double qm = a[ny - 1] - lam;
    if (abs_bits(qm) < pivbits) qm = -pivmin;
    ri = fast_rcp(qm);
    dm[(size_t)(ny - 1) * nm] = ri;
#pragma unroll 4
    for (int i = ny - 2; i >= 0; --i) {
      qm = fma(-b2[i], ri, a[i] - lam);
      if (abs_bits(qm) < pivbits) qm = -pivmin;
      const double gi = i > 0 ? fma(-b2[i - 1], dp[(size_t)(i - 1) * nm], qm) : qm;
      if (abs_bits(gi) < abs_bits(gam)) {
        gam = gi;
        r = i;
      }
      ri = fast_rcp(qm);
      dm[(size_t)i * nm] = ri;
    }
    // the vector out of r; its two end entries are kept apart (they alone carry D)
    z0 = r == 0 ? 1.0 : 0.0;
    z1 = r == ny - 1 ? 1.0 : 0.0;
    nint = r > 0 && r < ny - 1 ? 1.0 : 0.0;
    double z = 1.0;
#pragma unroll 4
    for (int i = r - 1; i >= 1; --i) {
      z *= -(b[i] * dp[(size_t)i * nm]);
      nint = fma(z, z, nint);
      dp[(size_t)i * nm] = z;
    }
    if (r > 0) {
      z0 = -(b[0] * dp[0]) * z;
      dp[0] = z0;
    }
    dp[(size_t)r * nm] = 1.0;
    z = 1.0;
#pragma unroll 4
    for (int i = r + 1; i < ny - 1; ++i) {
      z *= -(b[i - 1] * dm[(size_t)i * nm]);
      nint = fma(z, z, nint);
      dp[(size_t)i * nm] = z;
    }
    if (r < ny - 1) {
      z1 = -(b[ny - 2] * dm[(size_t)(ny - 1) * nm]) * z;
      dp[(size_t)(ny - 1) * nm] = z1;
    }
    const double delta = gam / fma(z0, z0, fma(z1, z1, nint));
    if (!(fabs(delta) < kCoarseMargin * gnorm)) break;      // NaN included
    // a step well above rounding says on which side of lambda the eigenvalue lies: for eigenvalue k the count is
    // then k or k + 1 (a count at the converged lambda alone could also be that of a close neighbour)
    if (fabs(delta) > 16.0 * atol) sure = neg == kf + k + (delta < 0.0 ? 1 : 0);
    lam += delta;
    if (!(fabs(lam - lam0) < 2 * kCoarseMargin * gnorm)) break;
    // a step at rounding level; a quarter of it while another factorisation is cheap
    if (fabs(delta) <= (it < 4 ? 0.25 : 1.0) * atol + 2.0 * DBL_EPSILON * fabs(lam)) {
      ok = sure && (neg == kf + k || neg == kf + k + 1);
      break;
    }
  }
  // v = D w, signed by its last entry
  const double v0 = z0 * r0s[q], v1 = z1 * r1s[q];
  const double sc = (v1 > 0.0 ? 1.0 : (v1 < 0.0 ? -1.0 : 0.0)) / sqrt(fma(v0, v0, fma(v1, v1, nint)));
  if (!ok || !isfinite(sc)) {
    fb.add(slice);
    return;
  }
  E[(size_t)slice * nm + k] = lam;
  double* out = Vsub + ((size_t)slice * nm + k) * ny;
  out[0] = sc * v0;
#pragma unroll 4
  for (int i = 1; i < ny - 1; ++i) out[i] = sc * dp[(size_t)i * nm];
  out[ny - 1] = sc * v1;
}

// One slice by FP64 multisection and one twisted factorisation per mode (one warp).
__device__ void bisect_slice(const double* __restrict__ me_y, const double* __restrict__ pot, double t0, int slice,
                             int nv, int nx, int ny, int nm, double* __restrict__ E, double* __restrict__ Vsub,
                             double* __restrict__ dplus, double* __restrict__ dminus, int* __restrict__ err) {
  extern __shared__ double smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SliceShared s = slice_shared(smem + (size_t)warp * slice_doubles(ny), ny);
  const double* m = me_y + (size_t)slice * ny;
  const double* V = pot + ((size_t)(slice / (nv * nx)) * nx + slice % nx) * ny;

  // 1. Ht's diagonal (rows 0 and ny-1 copy rows 1 and ny-2) and the symmetrised pairs.
  int bad = 0;
  for (int i = lane; i < ny; i += 32) {
    const int r = i == 0 ? 1 : (i == ny - 1 ? ny - 2 : i);
    const double lo = hop(t0, m[r - 1], m[r]), up = hop(t0, m[r + 1], m[r]);
    s.a[i] = -(lo + up) + V[r];
    if (!isfinite(s.a[i])) bad = 1;
    if (i < ny - 1) {
      const double U = i == 0 ? hop(t0, m[2], m[1]) : hop(t0, m[i + 1], m[i]);              // Ht(i, i+1)
      const double L = i + 1 == ny - 1 ? hop(t0, m[ny - 3], m[ny - 2]) : hop(t0, m[i], m[i + 1]);  // Ht(i+1, i)
      const double p = U * L;
      if (!(p > 0.0) || !isfinite(p)) bad = 1;
      s.b2[i] = p;
      s.b[i] = U < 0.0 ? -sqrt(p) : sqrt(p);
      s.rr[i] = sqrt(L / U);
    } else {
      s.b2[i] = 0.0;
      s.b[i] = 0.0;
      s.rr[i] = 1.0;
    }
    s.af[i] = (float)s.a[i];
    s.b2f[i] = (float)s.b2[i];
  }
  if (__any_sync(0xffffffffu, bad)) {
    if (lane == 0) atomicOr(err, 1);
    for (int k = lane; k < nm; k += 32) E[(size_t)slice * nm + k] = NAN;
    return;
  }
  __syncwarp();

  // Gershgorin interval of T and the pivot floor (LAPACK's dstebz convention).
  double glo = INFINITY, ghi = -INFINITY, bmax = 0.0;
  for (int i = lane; i < ny; i += 32) {
    const double rad = fabs(s.b[i]) + (i > 0 ? fabs(s.b[i - 1]) : 0.0);
    glo = fmin(glo, s.a[i] - rad);
    ghi = fmax(ghi, s.a[i] + rad);
    bmax = fmax(bmax, s.b2[i]);
  }
  for (int o = 16; o; o >>= 1) {
    glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
    ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
    bmax = fmax(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
  }
  const double gnorm = fmax(fabs(glo), fabs(ghi));
  const double pivmin = DBL_MIN * fmax(1.0, bmax);
  glo -= 2.0 * DBL_EPSILON * gnorm + 2.0 * pivmin;
  ghi += 2.0 * DBL_EPSILON * gnorm + 2.0 * pivmin;
  const double atol = DBL_EPSILON * gnorm;

  // 2. bisection of the candidates around zero
  const int n0 = __shfl_sync(0xffffffffu, lane == 0 ? sturm_count(s, ny, 0.0, pivmin) : 0, 0);
  const int c0 = max(0, n0 - nm), c1 = min(ny, n0 + nm), nc = c1 - c0;
  if (nc <= 16) {
    // multisection: candidate c on lanes [c g, c g + g); every lane of the warp takes part in
    // each step (the ballot), lanes past nc g and converged groups only vote 0
    const int g = 32 / nc, c = lane / g, j = lane % g;
    const bool mine = c < nc;
    const int k = c0 + (mine ? c : 0);
    const unsigned gmask = (g == 32 ? 0xffffffffu : ((1u << g) - 1u)) << (mine ? c * g : 0);
    // coarse FP32 multisection to ~1e-5 of the spectral radius (FP32 divisions are cheap)
    const float pivf = FLT_MIN * fmaxf(1.f, (float)bmax), ctol = 1e-5f * (float)gnorm;
    float flo = (float)glo, fhi = (float)ghi;
    for (int it = 0; it < 64; ++it) {
      const bool open = mine && fhi - flo > ctol;
      if (!__any_sync(0xffffffffu, open)) break;
      const float step = (fhi - flo) / (g + 1);
      const float p = flo + (j + 1) * step;
      const bool above = open && (p >= fhi || (p > flo && sturm_count32(s, ny, p, pivf) > k));
      const unsigned vote = __ballot_sync(0xffffffffu, above) & gmask;
      if (open) {
        const int jf = vote ? __ffs(vote) - 1 - c * g : g;
        const float nlo = jf == 0 ? flo : fmaxf(flo, flo + jf * step);
        const float nhi = jf == g ? fhi : fminf(fhi, flo + (jf + 1) * step);
        if (!(nlo > flo || nhi < fhi)) break;
        flo = nlo;
        fhi = nhi;
      }
    }
    // widen by a margin and confirm the bracket with FP64 counts (count(lo) <= k < count(hi)); a
    // bracket the FP32 counts got wrong falls back to the Gershgorin interval
    double lo = fmax(glo, (double)flo - 2e-5 * gnorm), hi = fmin(ghi, (double)fhi + 2e-5 * gnorm);
    {
      const bool chk = mine && j < 2;
      const int cnt = chk ? sturm_count(s, ny, j == 0 ? lo : hi, pivmin) : 0;
      const bool bad = chk && (j == 0 ? cnt > k : cnt <= k);
      if (__ballot_sync(0xffffffffu, bad) & gmask) {
        lo = glo;
        hi = ghi;
      }
    }
    for (int it = 0; it < 256; ++it) {
      const bool open = mine && hi - lo > atol + 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi));
      if (!__any_sync(0xffffffffu, open)) break;
      // lane j counts at p_j = lo + (j + 1) (hi - lo) / (g + 1); a point rounded onto or past an
      // end of the interval takes that end's known side (count(lo) <= k < count(hi))
      const double step = (hi - lo) / (g + 1);
      const double p = lo + (j + 1) * step;
      const bool above = open && (p >= hi || (p > lo && sturm_count(s, ny, p, pivmin) > k));
      const unsigned vote = __ballot_sync(0xffffffffu, above) & gmask;
      if (open) {
        // the first point of the group with more than k eigenvalues below it bounds from above
        const int jf = vote ? __ffs(vote) - 1 - c * g : g;
        const double nlo = jf == 0 ? lo : fmax(lo, lo + jf * step);
        const double nhi = jf == g ? hi : fmin(hi, lo + (jf + 1) * step);
        if (!(nlo > lo || nhi < hi)) {   // no progress at this resolution: the interval is final
          lo = hi = 0.5 * (lo + hi);
        } else {
          lo = nlo;
          hi = nhi;
        }
      }
    }
    if (mine && j == 0) s.lam[c] = 0.5 * (lo + hi);
  } else {
    for (int c = lane; c < nc; c += 32) {
      const int k = c0 + c;
      double lo = glo, hi = ghi;
      for (int it = 0; it < 256; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (!(hi - lo > atol + 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) || mid <= lo || mid >= hi) break;
        if (sturm_count(s, ny, mid, pivmin) > k) hi = mid;
        else lo = mid;
      }
      s.lam[c] = 0.5 * (lo + hi);
    }
  }
  __syncwarp();

  // 3. the nm of smallest magnitude: grow a window outwards from the sign change
  int lo = n0 - c0 - 1, hi = n0 - c0;
  for (int t = 0; t < nm; ++t) {
    if (hi < nc && (lo < 0 || fabs(s.lam[hi]) <= fabs(s.lam[lo]))) ++hi;
    else --lo;
  }
  const int first = lo + 1;

  // 4. eigenvectors, one lane per mode
  for (int k = lane; k < nm; k += 32) {
    const double lam = s.lam[first + k];
    E[(size_t)slice * nm + k] = lam;
    double* dp = dplus + (size_t)slice * ny * nm + k;    // [i][mode]
    double* dm = dminus + (size_t)slice * ny * nm + k;
    double q = guard(s.a[0] - lam, pivmin);
    dp[0] = q;
    for (int i = 1; i < ny; ++i) {
      q = guard(s.a[i] - lam - s.b2[i - 1] / q, pivmin);
      dp[(size_t)i * nm] = q;
    }
    double g = guard(s.a[ny - 1] - lam, pivmin);
    dm[(size_t)(ny - 1) * nm] = g;
    int r = ny - 1;
    double best = fabs(dp[(size_t)(ny - 1) * nm]);
    for (int i = ny - 2; i >= 0; --i) {
      g = guard(s.a[i] - lam - s.b2[i] / g, pivmin);
      dm[(size_t)i * nm] = g;
      const double gam = fabs(dp[(size_t)i * nm] + g - (s.a[i] - lam));
      if (gam < best) {
        best = gam;
        r = i;
      }
    }
    // w overwrites the top-down pivots: below r they are read just before being replaced
    dp[(size_t)r * nm] = 1.0;
    double w = 1.0;
    for (int i = r - 1; i >= 0; --i) {
      w = -(s.b[i] / dp[(size_t)i * nm]) * w;
      dp[(size_t)i * nm] = w;
    }
    w = 1.0;
    for (int i = r + 1; i < ny; ++i) {
      w = -(s.b[i - 1] / dm[(size_t)i * nm]) * w;
      dp[(size_t)i * nm] = w;
    }
    // v = D w, its norm and the sign of its last entry
    double d = 1.0, nrm = 0.0, last = 0.0;
    for (int i = 0; i < ny; ++i) {
      const double v = d * dp[(size_t)i * nm];
      nrm += v * v;
      last = v;
      d *= s.rr[i];
    }
    const double sc = (last > 0.0 ? 1.0 : (last < 0.0 ? -1.0 : 0.0)) / sqrt(nrm);
    if (!isfinite(sc)) atomicOr(err, 2);
    double* out = Vsub + ((size_t)slice * nm + k) * ny;
    d = 1.0;
    for (int i = 0; i < ny; ++i) {
      out[i] = sc * d * dp[(size_t)i * nm];
      d *= s.rr[i];
    }
  }
}

__global__ void __launch_bounds__(128) subband_bisect_kernel(const double* __restrict__ me_y,
                                                             const double* __restrict__ pot, double t0, int nv, int nx,
                                                             int ny, int nm, double* __restrict__ E,
                                                             double* __restrict__ Vsub, double* __restrict__ dplus,
                                                             double* __restrict__ dminus, int* __restrict__ err,
                                                             FallbackList fb) {
  const int nw = blockDim.x >> 5, n = *fb.count;
  for (int i = blockIdx.x * nw + (threadIdx.x >> 5); i < n; i += gridDim.x * nw) {
    bisect_slice(me_y, pot, t0, fb.list[i], nv, nx, ny, nm, E, Vsub, dplus, dminus, err);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256) subband_cleanup_kernel(double* __restrict__ Vsub, int batch, int nv, int nx,
                                                              int ny, int nm) {
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= (long long)batch * (nx - 1) * nm) return;
  const int b = (int)(warp / ((long long)(nx - 1) * nm));
  const int rem = (int)(warp % ((long long)(nx - 1) * nm));
  const int x = 1 + rem / nm, k = rem % nm;
  const size_t base = (size_t)b * nv * nx;                   // problem b, valley 1
  const double* v0 = Vsub + ((base + 0) * nm + k) * ny;      // slice 1
  double* v = Vsub + ((base + x) * nm + k) * ny;
  double dot = 0.0;
  for (int i = lane; i < ny; i += 32) dot += v0[i] * v[i];
  for (int o = 16; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (dot < -0.5)
    for (int i = lane; i < ny; i += 32) v[i] = -v[i];
}

__global__ void rcp_kernel(const double* __restrict__ x, double* __restrict__ y, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fast_rcp(x[i]);
}

size_t slice_smem(int ny) { return (size_t)slice_doubles(ny) * sizeof(double); }

int warps_per_block(int ny) {
  int w = 4;
  while (w > 1 && (size_t)w * slice_smem(ny) > 160 * 1024) --w;
  return w;
}

}  // namespace

struct wg_subbands {
  int batch = 0, nv = 0, nx = 0, ny = 0, nm = 0;
  cudaStream_t stream = nullptr;
  double *me_y = nullptr, *V = nullptr, *E = nullptr, *Vsub = nullptr, *dp = nullptr, *dm = nullptr;
  int* err = nullptr;
  int* kfirst = nullptr;     // [slices] index of the first eigenvalue taken, -1: left to the bisection
  int* fallback = nullptr;   // count, flag [slices], list [slices]
  std::string msg;
};

extern "C" {

int wg_debug_rcp(const double* x, double* y, long long n) {
  if (!x || !y || n < 1 || n > (1ll << 28)) return WG_ERR_ARG;
  double* d = nullptr;
  const size_t sz = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&d, 2 * sz);
  if (e == cudaSuccess) e = cudaMemcpy(d, x, sz, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    rcp_kernel<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, d + n, sz, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? WG_OK : WG_ERR_CUDA;
}

int wg_subbands_create(int batch, int n_valleys, int nx, int ny, int n_modes, wg_subbands** out) {
  if (!out) return WG_ERR_ARG;
  *out = nullptr;
  if (batch < 1 || n_valleys < 1 || nx < 1 || ny < 3 || ny > kMaxNy || n_modes < 1 || n_modes > kMaxModes ||
      n_modes > ny || (long long)batch * n_valleys * nx > (1LL << 30))
    return WG_ERR_ARG;
  wg_subbands* h = new wg_subbands;
  h->batch = batch;
  h->nv = n_valleys;
  h->nx = nx;
  h->ny = ny;
  h->nm = n_modes;
  const size_t slices = (size_t)batch * n_valleys * nx;
  cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&h->me_y, slices * ny * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->V, (size_t)batch * nx * ny * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->E, slices * n_modes * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->Vsub, slices * n_modes * ny * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->dp, slices * n_modes * ny * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->dm, slices * n_modes * ny * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->err, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(h->err, 0, sizeof(int));
  if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);   // the solves' streams do not wait for it
  if (e == cudaSuccess) e = cudaMalloc(&h->kfirst, slices * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&h->fallback, (2 * slices + 1) * sizeof(int));
  // the largest block's limit: it belongs to the kernel, and a later handle must not lower it for this one
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(subband_bisect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
  if (e != cudaSuccess) {
    wg_subbands_destroy(h);
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? WG_ERR_OOM : WG_ERR_CUDA;
  }
  *out = h;
  return WG_OK;
}

int wg_subbands_destroy(wg_subbands* h) {
  if (!h) return WG_OK;
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (double* p : {h->me_y, h->V, h->E, h->Vsub, h->dp, h->dm})
    if (p) cudaFree(p);
  for (int* p : {h->err, h->kfirst, h->fallback})
    if (p) cudaFree(p);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return WG_OK;
}

const char* wg_subbands_last_error(const wg_subbands* h) { return h ? h->msg.c_str() : "null handle"; }

int wg_subbands_solve_device(wg_subbands* h, double dy_nm, const double* me_y, const double* V, double* E,
                             double* Vsub, void* stream) {
  if (!h || !me_y || !V || !E || !Vsub || !(dy_nm > 0.0)) return WG_ERR_ARG;
  cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
  const double hb = 6.626e-34 / 2 / M_PI;
  const double t0 = hb * hb / 2 / (9.109e-31 * dy_nm * dy_nm * 1.602e-19 * 1e-18);   // eval_transversal_Hamiltonian.m:20
  const int slices = h->batch * h->nv * h->nx, wpb = warps_per_block(h->ny);
  const FallbackList fb{h->fallback, h->fallback + 1, h->fallback + 1 + slices};
  cudaMemsetAsync(h->fallback, 0, (1 + (size_t)slices) * sizeof(int), st);
  subband_coarse_kernel<<<(slices + 3) / 4, 128, 4 * coarse_floats(h->ny) * sizeof(float), st>>>(
      me_y, V, (float)t0, slices, h->nv, h->nx, h->ny, h->nm, E, h->kfirst, t0, h->dp, h->dm, fb);
  const int sl = refine_slices(h->ny, h->nm);
  subband_refine_kernel<<<(slices + sl - 1) / sl, 32, sl * refine_doubles(h->ny) * sizeof(double), st>>>(
      me_y, V, t0, slices, h->nv, h->nx, h->ny, h->nm, sl, E, Vsub, h->dp, h->dm, h->kfirst, fb);
  subband_bisect_kernel<<<std::min((slices + wpb - 1) / wpb, 608), 32 * wpb, wpb * slice_smem(h->ny), st>>>(
      me_y, V, t0, h->nv, h->nx, h->ny, h->nm, E, Vsub, h->dp, h->dm, h->err, fb);
  if (h->nx > 1) {
    const long long warps = (long long)h->batch * (h->nx - 1) * h->nm;
    subband_cleanup_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(Vsub, h->batch, h->nv, h->nx,
                                                                                  h->ny, h->nm);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    h->msg = cudaGetErrorString(e);
    return WG_ERR_CUDA;
  }
  return WG_OK;
}

int wg_subbands_status(wg_subbands* h, void* stream) {
  if (!h) return WG_ERR_ARG;
  cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
  int flag = 0;
  cudaError_t e = cudaMemcpyAsync(&flag, h->err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(h->err, 0, sizeof(int), st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    h->msg = cudaGetErrorString(e);
    return WG_ERR_CUDA;
  }
  if (flag & 1) {
    h->msg = "non-finite Hamiltonian entry or non-positive off-diagonal product (masses must be positive)";
    return WG_ERR_NUMERIC;
  }
  if (flag & 2) {
    h->msg = "eigenvector with a zero or non-finite last entry";
    return WG_ERR_NUMERIC;
  }
  return WG_OK;
}

int wg_subbands_solve(wg_subbands* h, double dy_nm, const double* me_y, const double* V, double* E, double* Vsub) {
  if (!h || !me_y || !V || !E || !Vsub || !(dy_nm > 0.0)) return WG_ERR_ARG;
  const size_t slices = (size_t)h->batch * h->nv * h->nx;
  for (size_t i = 0; i < slices * h->ny; ++i)
    if (!(me_y[i] > 0.0) || !std::isfinite(me_y[i])) {
      h->msg = "effective masses must be positive and finite";
      return WG_ERR_ARG;
    }
  for (size_t i = 0; i < (size_t)h->batch * h->nx * h->ny; ++i)
    if (!std::isfinite(V[i])) {
      h->msg = "potential must be finite";
      return WG_ERR_ARG;
    }
  cudaError_t e = cudaMemcpyAsync(h->me_y, me_y, slices * h->ny * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->V, V, (size_t)h->batch * h->nx * h->ny * sizeof(double), cudaMemcpyHostToDevice,
                        h->stream);
  if (e != cudaSuccess) {
    h->msg = cudaGetErrorString(e);
    return WG_ERR_CUDA;
  }
  int rc = wg_subbands_solve_device(h, dy_nm, h->me_y, h->V, h->E, h->Vsub, h->stream);
  if (rc != WG_OK) return rc;
  e = cudaMemcpyAsync(E, h->E, slices * h->nm * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(Vsub, h->Vsub, slices * h->nm * h->ny * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  if (e != cudaSuccess) {
    h->msg = cudaGetErrorString(e);
    return WG_ERR_CUDA;
  }
  return wg_subbands_status(h, h->stream);
}

int wg_subbands_buffers(wg_subbands* h, double** me_y, double** V, double** E, double** Vsub) {
  if (!h) return WG_ERR_ARG;
  if (me_y) *me_y = h->me_y;
  if (V) *V = h->V;
  if (E) *E = h->E;
  if (Vsub) *Vsub = h->Vsub;
  return WG_OK;
}

}  // extern "C"
