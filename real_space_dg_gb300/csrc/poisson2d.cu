// 2D Poisson step of the Full-2D Gummel loop on the device (sm_103a).
//
// The reference's electrostatic step (RTD/make_RTD_poisson_step.m:44-54):
//   n   = project_DG_density_RTD(nDG)         exact DG integrals over the dual volumes
//                                             (RTD/project_DG_density_RTD.m:16-31)
//   phi = solve_Poisson2D_rtd(M, n, phi0)     the direct or approximate-Newton update on the
//                                             unique nodes (RTD/solve_Poisson2D_rtd.m:64-131)
// with M the 5-point div(eps grad) operator of RTD/eval_Poisson2D_rtd.m:107-188 (harmonic-mean
// faces, half control volumes at free X ends and non-periodic Y ends, Dirichlet identity rows,
// Y endpoints identified when periodic).
//
// Unique nodes k = ix + iy nx (x fastest, MATLAB's order), iy < nu (nu = Ny - 1 when periodic).
// The update solves J d = -F(free) with J = A_ff (direct) or A_ff - diag(q^2 n / (kB T)) (Newton),
// ordered by x columns: J is block tridiagonal, the column blocks D (the Y stencil, a ring when periodic, plus
// the diagonal) coupled to the neighbour columns by diagonal matrices L, U (the X faces).  J is diagonally dominant
// and so are the Schur complements below, so blocks are eliminated without pivoting; Dirichlet nodes stay in as
// identity rows with a zero right-hand side.
//
// Block cyclic reduction over x: level by level every second remaining column is eliminated,
//   D_c' = D_c - L_c D_l^-1 U_l - U_c D_r^-1 L_r,  L_c' = -L_c D_l^-1 L_l,  U_c' = -U_c D_r^-1 U_r,
//   r_c' = r_c - L_c D_l^-1 r_l - U_c D_r^-1 r_r            (l, r: the eliminated neighbours of kept column c),
// all columns of a level at once, one block each (poisson2d_reduce_kernel), then the levels are substituted back.
// log2(nx) + 1 dependent steps instead of a sweep over nx columns: the sweep (one warp per bias point) was
// a chain of nx inversions, 20 us each.  Measured with a 361 x 13 periodic grid, projection and update of 16 bias points:
// 7.4 ms with the sweep, 0.32 ms here (one point, 97 x 11: 1.9 -> 0.12 ms).
// Every reduction over nodes has a fixed order that does not depend on the batch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>
#include <vector>

#include "recip.cuh"
#include "wigner_gb300.h"

using wg::fast_rcp;

namespace {

constexpr double kQ = 1.602176634e-19;
constexpr double kKB = 1.380649e-23;
constexpr double kEps0 = 8.8541878128e-12;

struct P2Dev {
  int nx, ny, nu, periodic, batch;
  const unsigned char* fixed;     // [nu nx]
  const double *cxm, *cxp, *cym, *cyp, *diag;   // stencil of the free rows (0 on fixed rows)
  const double* net;              // Nd - Na [nu nx]
  const double *vx, *vy;          // control-volume widths for the charge diagnostics [nx], [nu]
  // projection (optional)
  int ndx, ndy;
  const int *tx_rp, *tx_col, *ty_rp, *ty_col;
  const double *tx_val, *ty_val, *wx, *wy, *srcx, *srcy;
};

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// of non-negative values, NaN ignored: as integers, which their bit patterns are ordered like
__device__ __forceinline__ double warp_max(double v) {
  long long u = __double_as_longlong(v);
  if (u > 0x7ff0000000000000ll) u = 0;
  for (int o = 16; o; o >>= 1) {
    const long long t = __shfl_xor_sync(0xffffffffu, u, o);
    u = t > u ? t : u;
  }
  return __longlong_as_double(u);
}

// Sums of v[0 .. NS) and maxima of the non-negative v[NS .. N) over a block of 256 threads, fixed order; out[i] is
// written by one thread each, without a barrier after it.
template <int N, int NS>
__device__ void block_reduce(const double (&v)[N], double (*red)[8], double* out, int stride) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    double t = v[i];
    if (i < NS) t = warp_sum(t);
    else t = warp_max(t);
    if (lane == 0) red[i][warp] = t;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    const int i = threadIdx.x;
    double t = red[i][0];
    for (int q = 1; q < 8; ++q) t = i < NS ? t + red[i][q] : fmax(t, red[i][q]);
    out[(size_t)i * stride] = t;
  }
}

// Buffers of one step (the B problems of a group, launch_step): n, v, F [B][nun]; r, y, d [B][nx][NU]; the blocks of
// the reduction and the block partials of the reductions over nodes.
struct P2Work {
  double *n, *v, *F, *r, *y, *d;
  double *D, *L, *U;      // [B][nx / 2][NU][NU]: the odd columns' blocks of the current level
  double *XL, *XU;        // [B][nx / 2][NU][NU]: D^-1 L and D^-1 U of the columns eliminated above level 0
  double* Dinv;           // [B][(nx + 1) / 2][NU][NU]: D^-1 of the even columns (eliminated at level 0)
  double* part;           // [B][kP2Part][blocks]
  int* count;             // [B] tickets of the last step kernel (zero between launches)
};
constexpr int kP2Threads = 256, kP2Part = 14;

// 1. The density on the unique nodes (DG integrals over the dual volumes, or given), v = phi0 with the contacts
// set, F = A v - charge, r = -F on the free nodes, and the block partials of the scale and the integrals.
__global__ void __launch_bounds__(kP2Threads) poisson2d_assemble_kernel(P2Dev P, P2Work w, int NU,
                                                                        const double* __restrict__ src, int src_is_dg,
                                                                        const double* __restrict__ phi0,
                                                                        const double* __restrict__ bc) {
  __shared__ double red[6][8];
  const int b = blockIdx.y, nx = P.nx, nu = P.nu, nun = nu * nx;
  const size_t full = (size_t)nx * P.ny;
  src += (size_t)b * (src_is_dg ? (size_t)P.ndx * P.ndy : full);
  phi0 += (size_t)b * full;
  bc += (size_t)b * nun;
  const int k = blockIdx.x * kP2Threads + threadIdx.x;
  double src_int = 0.0, tgt_int = 0.0, m_qn = 0.0, m_qnet = 0.0, m_av = 0.0, m_f = 0.0;
  auto vat = [&](int q) { return P.fixed[q] ? bc[q] : phi0[q]; };
  if (k < nun) {
    const int ix = k % nx, iy = k / nx;
    double nk;
    if (src_is_dg) {
      double acc = 0.0;
      for (int p = P.tx_rp[ix]; p < P.tx_rp[ix + 1]; ++p) {
        const double* row = src + P.tx_col[p];
        double s = 0.0;
        for (int q = P.ty_rp[iy]; q < P.ty_rp[iy + 1]; ++q) s += P.ty_val[q] * row[(size_t)P.ty_col[q] * P.ndx];
        acc += P.tx_val[p] * s;
      }
      tgt_int = acc;
      nk = acc / (P.wx[ix] * P.wy[iy]);
    } else {
      nk = src[k];
    }
    const double v = vat(k);
    double av = v;
    const bool fx = P.fixed[k];
    if (!fx) {
      av = P.diag[k] * v;
      if (ix > 0) av += P.cxm[k] * vat(k - 1);
      if (ix < nx - 1) av += P.cxp[k] * vat(k + 1);
      if (iy > 0 || P.periodic) av += P.cym[k] * vat((iy > 0 ? iy - 1 : nu - 1) * nx + ix);
      if (iy < nu - 1 || P.periodic) av += P.cyp[k] * vat((iy < nu - 1 ? iy + 1 : 0) * nx + ix);
    }
    const double f = av - kQ * (nk - P.net[k]);
    if (!fx) {
      m_qn = fabs(kQ * nk);
      m_qnet = fabs(kQ * P.net[k]);
      m_av = fabs(av);
      m_f = fabs(f);
    }
    const size_t g = (size_t)b * nun + k;
    w.n[g] = nk;
    w.v[g] = v;
    w.F[g] = f;
    w.r[((size_t)b * nx + ix) * NU + iy] = fx ? 0.0 : -f;
  }
  // rows nu .. NU-1 of every column are identity padding with a zero right-hand side
  for (int q = k; q < nx * (NU - nu); q += gridDim.x * kP2Threads)
    w.r[((size_t)b * nx + q % nx) * NU + nu + q / nx] = 0.0;
  if (src_is_dg)
    for (int e = k; e < P.ndx * P.ndy; e += gridDim.x * kP2Threads)
      src_int += P.srcx[e % P.ndx] * src[e] * P.srcy[e / P.ndx];
  const double v6[6] = {src_int, tgt_int, m_qn, m_qnet, m_av, m_f};
  block_reduce<6, 2>(v6, red, w.part + (size_t)b * kP2Part * gridDim.x + blockIdx.x, gridDim.x);
}

// Entry (i, j) of column c's diagonal block of J; rows of fixed nodes (and the padding) are identity rows, and
// couplings to fixed nodes are dropped (their update is zero).
__device__ __forceinline__ double block_entry(const P2Dev& P, const double* __restrict__ n, int newton, double q_kt,
                                              int c, int i, int j) {
  if (i >= P.nu || j >= P.nu) return i == j ? 1.0 : 0.0;
  const int k = c + i * P.nx;
  if (P.fixed[k]) return i == j ? 1.0 : 0.0;
  if (i == j) return P.diag[k] - (newton ? q_kt * n[k] : 0.0);
  if (P.fixed[c + j * P.nx]) return 0.0;
  const int jm = i > 0 ? i - 1 : (P.periodic ? P.nu - 1 : -1);
  const int jp = i < P.nu - 1 ? i + 1 : (P.periodic ? 0 : -1);
  return (j == jm ? P.cym[k] : 0.0) + (j == jp ? P.cyp[k] : 0.0);
}
// Couplings of row i of column c to the same row of the columns c - 1 and c + 1.
__device__ __forceinline__ double left_entry(const P2Dev& P, int c, int i) {
  const int k = c + i * P.nx;
  return i < P.nu && c > 0 && !P.fixed[k] && !P.fixed[k - 1] ? P.cxm[k] : 0.0;
}
__device__ __forceinline__ double right_entry(const P2Dev& P, int c, int i) {
  const int k = c + i * P.nx;
  return i < P.nu && c < P.nx - 1 && !P.fixed[k] && !P.fixed[k + 1] ? P.cxp[k] : 0.0;
}

// 2a. Level 0: D^-1 and y = D^-1 r of every even column (one block each).
// 2b. Level l >= 1, s = 2^l: the columns c_k = (k + 1) s - 1, k < K = nx / s, are still there.  The block of c_k first
// folds the neighbours c_k -+ s/2 that the level before eliminated into D, L, U and r (level 1: the couplings
// are diagonal and come from the stencil), then an even k eliminates: [X_L X_U y] = D^-1 [L U r]; an odd k stores
// the folded blocks.  Thread (i, q) keeps row i, columns q + t TPR of the augmented matrix in registers.
//
// A warp's FP64 instruction takes its SM quarter's pipe for 64 cycles and returns after as many, so a block has few warps, and
// what counts in a latter level, where a handful of blocks run, is instructions per pivot: CPT updates, one
// product, and the reciprocal (4, by the pivot's warp alone).  Both neighbours in one block (eliminating a shared one twice)
// and 1 / x by division took 93, 82 and 44 us at levels 0, 1 and 2 of 16 bias points on 361 columns of 12 rows, 436 us for
// the whole step; here it takes 324 us.
// Columns per thread by width, whole step in us, 16 points of 361 columns and one of 97 (chosen first): 4 rows 122 and 78
// with 4 columns, 123 and 81 with 3; 8 rows 192 and 91 with 3, 203 and 109 with 4; 12 rows 324 and 122, 336 and 138; 16 rows 523
// and 157, 538 and 168; 24 rows 1,325 and 369 with 8, 1,419 and 338 with 4; 32 rows 2,896 and 636, 3,541 and 723.  That is 1,
// 3, 5, 9, 8 and 13 warps a block, one to six at level 0 up to 16 rows.
template <int NU, int NB>
struct ReduceShape {
  static constexpr int W = NB * NU + 1;                       // augmented width: NB blocks and r
  static constexpr int CPT = NU >= 24 ? 8 : NU >= 8 ? 3 : 4;   // columns per thread
  static constexpr int TPR = (W + CPT - 1) / CPT;             // threads per row
  static constexpr int THREADS = (NU * TPR + 31) / 32 * 32;
};

// [D | rest] -> D^-1 rest in registers, no pivoting; dg[i]: 1 / the pivot of row i.
template <int NU, int NB>
__device__ void eliminate(double (&a)[ReduceShape<NU, NB>::CPT], int i, int q, bool on,
                          double (*rowb)[ReduceShape<NU, NB>::W], double (*colb)[NU], double* dg) {
  using S = ReduceShape<NU, NB>;
#pragma unroll
  for (int p = 0; p < NU; ++p) {
    const int bf = p & 1;
    if (on) {
      if (q == p % S::TPR) {
        colb[bf][i] = a[p / S::TPR];
        if (i == p) dg[p] = fast_rcp(a[p / S::TPR]);
      }
      if (i == p)
#pragma unroll
        for (int t = 0; t < S::CPT; ++t)
          if (q + t * S::TPR < S::W) rowb[bf][q + t * S::TPR] = a[t];
    }
    __syncthreads();
    if (on && i != p) {
      const double f = -colb[bf][i] * dg[p];
#pragma unroll
      for (int t = 0; t < S::CPT; ++t)
        if (p < (t + 1) * S::TPR - 1 && q + t * S::TPR < S::W)   // columns up to p are done with
          a[t] = fma(f, rowb[bf][q + t * S::TPR], a[t]);
    }
  }
  if (on) {
    const double d = dg[i];
#pragma unroll
    for (int t = 0; t < S::CPT; ++t) a[t] *= d;
  }
}

template <int NU>
__global__ void __launch_bounds__(ReduceShape<NU, 2>::THREADS)
    poisson2d_invert_kernel(P2Dev P, P2Work w, int newton, double q_kt) {
  using S = ReduceShape<NU, 2>;
  __shared__ double rowb[2][S::W], colb[2][NU], dg[NU];
  const int b = blockIdx.y, nx = P.nx, c = 2 * blockIdx.x;
  const int i = threadIdx.x / S::TPR, q = threadIdx.x % S::TPR;
  const bool on = i < NU;
  const double* n = w.n + (size_t)b * P.nu * nx;
  double a[S::CPT];
#pragma unroll
  for (int t = 0; t < S::CPT; ++t) {
    const int j = q + t * S::TPR;
    a[t] = !on || j >= S::W ? 0.0
                            : j < NU ? block_entry(P, n, newton, q_kt, c, i, j)
                                     : j < 2 * NU ? (j - NU == i ? 1.0 : 0.0) : w.r[((size_t)b * nx + c) * NU + i];
  }
  eliminate<NU, 2>(a, i, q, on, rowb, colb, dg);
  if (on)
#pragma unroll
    for (int t = 0; t < S::CPT; ++t) {
      const int j = q + t * S::TPR;
      if (j == 2 * NU) w.y[((size_t)b * nx + c) * NU + i] = a[t];
      else if (j >= NU && j < 2 * NU)
        w.Dinv[(((size_t)b * ((nx + 1) / 2) + blockIdx.x) * NU + i) * NU + j - NU] = a[t];
    }
}

template <int NU, bool FIRST>
__global__ void __launch_bounds__(ReduceShape<NU, 3>::THREADS)
    poisson2d_reduce_kernel(P2Dev P, P2Work w, int newton, double q_kt, int s) {
  using S = ReduceShape<NU, 3>;
  constexpr int BB = NU * NU, CPT = S::CPT, TPR = S::TPR;
  __shared__ double rowb[2][S::W], colb[2][NU], dg[NU];
  const int b = blockIdx.y, nx = P.nx, nh = nx / 2, k = blockIdx.x;
  const int c = (k + 1) * s - 1, cl = c - s / 2, cr = c + s / 2;
  const bool has_r = cr < nx;
  const int i = threadIdx.x / TPR, q = threadIdx.x % TPR;
  const bool on = i < NU;
  const double* n = w.n + (size_t)b * P.nu * nx;
  double* r = w.r + (size_t)b * nx * NU;
  double* y = w.y + (size_t)b * nx * NU;
  auto blk = [&](double* base, int col) { return base + ((size_t)b * nh + col / 2) * BB; };   // col is odd here
  // 1. fold: D -= L XU_l + U XL_r, L = -L XL_l, U = -U XU_r, r -= L y_l + U y_r
  // up to 16 rows the six blocks and the products L XL_l, L XU_l, U XL_r, U XU_r, L y_l, U y_r go through shared
  // memory: one round of loads, and every lane of the products' FMAs is used
  constexpr bool STAGED = !FIRST && NU <= 16;
  constexpr int PR = 4 * BB + 2 * NU;
  __shared__ double sb[STAGED ? 6 * BB + 2 * NU : 1], pr_s[STAGED ? PR : 1];
  if constexpr (STAGED) {
    const double* src[6] = {blk(w.L, c), blk(w.U, c), blk(w.XL, cl), blk(w.XU, cl),
                            has_r ? blk(w.XL, cr) : nullptr, has_r ? blk(w.XU, cr) : nullptr};
#pragma unroll
    for (int m = 0; m < 6; ++m)
      for (int e = threadIdx.x; e < BB; e += S::THREADS) sb[m * BB + e] = src[m] ? src[m][e] : 0.0;
    for (int e = threadIdx.x; e < 2 * NU; e += S::THREADS)
      sb[6 * BB + e] = e < NU ? y[(size_t)cl * NU + e] : (has_r ? y[(size_t)cr * NU + e - NU] : 0.0);
    __syncthreads();
    for (int e = threadIdx.x; e < PR; e += S::THREADS) {
      // product m of row o / NU, column o % NU; the last 2 NU are the vectors
      const int m = e / BB, o = m < 4 ? e % BB : 0, v = e - 4 * BB;
      const double* cf = sb + (m < 4 ? (m < 2 ? 0 : BB) + o / NU * NU : (v < NU ? 0 : BB) + v % NU * NU);
      const double* xc = sb + (m < 4 ? (2 + m) * BB + o % NU : 6 * BB + v / NU * NU);
      const int st = m < 4 ? NU : 1;
      double v0 = 0.0, v1 = 0.0;
#pragma unroll
      for (int h = 0; h < NU; h += 2) {
        v0 = fma(cf[h], xc[h * st], v0);
        v1 = fma(cf[h + 1], xc[(h + 1) * st], v1);
      }
      pr_s[e] = v0 + v1;
    }
    __syncthreads();
  }
  double a[CPT];
#pragma unroll
  for (int t = 0; t < CPT; ++t) {
    const int j = q + t * TPR, jb = j / NU, jc = j % NU;   // block 0 D, 1 L, 2 U, 3 r
    a[t] = 0.0;
    if (!on || j >= S::W) continue;
    if (FIRST) {
      const double l = left_entry(P, c, i), u = has_r ? right_entry(P, c, i) : 0.0;
      if (jb == 3) {
        a[t] = r[(size_t)c * NU + i] - l * y[(size_t)cl * NU + i];
        if (has_r) a[t] = fma(-u, y[(size_t)cr * NU + i], a[t]);
        continue;
      }
      const double* dl = w.Dinv + ((size_t)b * ((nx + 1) / 2) + cl / 2) * BB + i * NU + jc;
      const double gl = jb < 2 ? -l * dl[0] : 0.0, gr = jb != 1 && has_r ? -u * dl[BB] : 0.0;
      if (jb == 0) {
        a[t] = fma(gl, right_entry(P, cl, jc), block_entry(P, n, newton, q_kt, c, i, jc));
        if (has_r) a[t] = fma(gr, left_entry(P, cr, jc), a[t]);
      } else if (jb == 1) {
        a[t] = gl * left_entry(P, cl, jc);
      } else if (has_r) {
        a[t] = gr * right_entry(P, cr, jc);
      }
    } else if constexpr (STAGED) {
      const int o = i * NU + jc;
      if (jb == 0) a[t] = blk(w.D, c)[o] - (pr_s[BB + o] + pr_s[2 * BB + o]);
      else if (jb == 1) a[t] = -pr_s[o];
      else if (jb == 2) a[t] = -pr_s[3 * BB + o];
      else a[t] = r[(size_t)c * NU + i] - (pr_s[4 * BB + i] + pr_s[4 * BB + NU + i]);
    } else {
      const double *Lc = blk(w.L, c) + i * NU, *Uc = blk(w.U, c) + i * NU;
      // the factors of L and of U in this column (r: vectors)
      const double *pl = jb == 3 ? y + (size_t)cl * NU : jb == 2 ? nullptr : blk(jb == 0 ? w.XU : w.XL, cl) + jc;
      const double *pr = !has_r || jb == 1 ? nullptr
                                           : jb == 3 ? y + (size_t)cr * NU : blk(jb == 0 ? w.XL : w.XU, cr) + jc;
      const int st = jb == 3 ? 1 : NU;
      double v = jb == 0 ? blk(w.D, c)[i * NU + jc] : jb == 3 ? r[(size_t)c * NU + i] : 0.0;
      if (pl)
#pragma unroll 4
        for (int m = 0; m < NU; ++m) v = fma(-Lc[m], pl[m * st], v);
      if (pr)
#pragma unroll 4
        for (int m = 0; m < NU; ++m) v = fma(-Uc[m], pr[m * st], v);
      a[t] = v;
    }
  }
  const bool keep = k & 1;   // stays: the next level folds and eliminates it or keeps it on
  if (keep) __syncthreads();   // the block's old L and U have been read
  else eliminate<NU, 3>(a, i, q, on, rowb, colb, dg);   // 2.
  if (!on) return;
#pragma unroll
  for (int t = 0; t < CPT; ++t) {
    const int j = q + t * TPR, jb = j / NU, o = i * NU + j % NU;
    if (jb == 0 && keep) blk(w.D, c)[o] = a[t];
    else if (jb == 1) blk(keep ? w.L : w.XL, c)[o] = a[t];
    else if (jb == 2) blk(keep ? w.U : w.XU, c)[o] = a[t];
    else if (j == 3 * NU) (keep ? r : y)[(size_t)c * NU + i] = a[t];
  }
}

// 3. Back substitution of levels hi .. lo (2^lo = s_lo): d_c = y_c - XL_c d_{c-s} - XU_c d_{c+s}.  With
// grouped == 0 the block takes every column of these levels; otherwise lo == 0 and block x takes the columns of
// [8 x, 8 x + 8), whose ends above level 2 are known, in levels 2, 1, 0.  Eight threads per row of a column.
template <int NU>
__global__ void __launch_bounds__(kP2Threads) poisson2d_back_kernel(P2Dev P, P2Work w, int s_hi, int s_lo,
                                                                    int grouped) {
  constexpr int LN = 8;
  const int b = blockIdx.y, nx = P.nx, nh = nx / 2, sub = threadIdx.x % LN;
  const double* y = w.y + (size_t)b * nx * NU;
  double* d = w.d + (size_t)b * nx * NU;
  const int c0 = grouped ? 8 * blockIdx.x : 0, c1 = grouped ? min(nx, c0 + 8) : nx;
  for (int s = s_hi; s >= s_lo; s /= 2) {
    // columns eliminated at stride s: c = s - 1 + 2 s m
    const int cnt = c1 - c0 >= s ? (c1 - c0 - s) / (2 * s) + 1 : 0;
    for (int e0 = 0; e0 < cnt * NU; e0 += kP2Threads / LN) {
      const int e = e0 + threadIdx.x / LN;
      const bool on = e < cnt * NU;
      const int c = c0 + s - 1 + 2 * s * ((on ? e : 0) / NU), i = (on ? e : 0) % NU;
      const bool hl = c - s >= 0, hr = c + s < nx;
      const double* dl = d + (size_t)(c - s) * NU;
      const double* dr = d + (size_t)(c + s) * NU;
      double v = 0.0;
      if (on) {
        if (s == 1) {
          const double* m = w.Dinv + (((size_t)b * ((nx + 1) / 2) + c / 2) * NU + i) * NU;
#pragma unroll
          for (int j = sub; j < NU; j += LN) {
            double t = 0.0;
            if (hl) t = left_entry(P, c, j) * dl[j];
            if (hr) t = fma(right_entry(P, c, j), dr[j], t);
            v = fma(m[j], t, v);
          }
        } else {
          const size_t o = (((size_t)b * nh + c / 2) * NU + i) * NU;
#pragma unroll
          for (int j = sub; j < NU; j += LN) {
            if (hl) v = fma(w.XL[o + j], dl[j], v);
            if (hr) v = fma(w.XU[o + j], dr[j], v);
          }
        }
      }
#pragma unroll
      for (int o = LN / 2; o; o /= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (on && sub == 0) d[(size_t)c * NU + i] = y[(size_t)c * NU + i] - v;
    }
    __syncthreads();
  }
}

// 4. The linear residual J d + F, the update, the residual after it, the diagnostics, and phi and the density
// on the full grid (the duplicate Y column when periodic).  The last block of a problem adds the partials.
__global__ void __launch_bounds__(kP2Threads) poisson2d_finish_kernel(P2Dev P, P2Work w, int NU,
                                                                      const double* __restrict__ phi0, int newton,
                                                                      double q_kt, double alpha,
                                                                      double* __restrict__ phi,
                                                                      double* __restrict__ density,
                                                                      wg_poisson2d_info* __restrict__ info) {
  __shared__ double red[8][8], all[kP2Part];
  __shared__ int last;
  const int b = blockIdx.y, nx = P.nx, nu = P.nu, nun = nu * nx;
  const size_t full = (size_t)nx * P.ny;
  const double* n = w.n + (size_t)b * nun;
  const double* v = w.v + (size_t)b * nun;
  const double* F = w.F + (size_t)b * nun;
  const double* d = w.d + (size_t)b * nx * NU;
  const int k = blockIdx.x * kP2Threads + threadIdx.x;
  double m_lin = 0.0, m_d = 0.0, e2 = 0.0, m_after = 0.0, qnet = 0.0, qabs_net = 0.0, qabs_n = 0.0, bad = 0.0;
  if (k < nun) {
    const int ix = k % nx, iy = k / nx;
    auto dat = [&](int x, int yy) { return P.fixed[x + yy * nx] ? 0.0 : d[(size_t)x * NU + yy]; };
    const double t = dat(ix, iy), up = P.fixed[k] ? v[k] : v[k] + alpha * t;
    const double ch = kQ * (n[k] - P.net[k]);
    if (!P.fixed[k]) {
      double jd = P.diag[k] * t, au = P.diag[k] * up;
      auto nbr = [&](double cf, int x, int yy) {
        const double dn = dat(x, yy);
        jd += cf * dn;
        au += cf * (P.fixed[x + yy * nx] ? v[x + yy * nx] : v[x + yy * nx] + alpha * dn);
      };
      if (ix > 0) nbr(P.cxm[k], ix - 1, iy);
      if (ix < nx - 1) nbr(P.cxp[k], ix + 1, iy);
      if (iy > 0 || P.periodic) nbr(P.cym[k], ix, iy > 0 ? iy - 1 : nu - 1);
      if (iy < nu - 1 || P.periodic) nbr(P.cyp[k], ix, iy < nu - 1 ? iy + 1 : 0);
      m_lin = fabs(jd - (newton ? q_kt * n[k] * t : 0.0) + F[k]);
      m_d = fabs(t);
      const double dd = up - phi0[(size_t)b * full + k];
      e2 = dd * dd;
      m_after = fabs(au - ch);
    }
    const double vol = P.vx[ix] * P.vy[iy];
    qnet = vol * ch;
    qabs_net = vol * fabs(P.net[k]);
    qabs_n = vol * fabs(n[k]);
    bad = isfinite(up) ? 0.0 : 1.0;
    phi[b * full + k] = up;
    density[b * full + k] = n[k];
    if (P.periodic && iy == 0) {
      phi[b * full + (size_t)nu * nx + ix] = up;
      density[b * full + (size_t)nu * nx + ix] = n[k];
    }
  }
  double* part = w.part + (size_t)b * kP2Part * gridDim.x;   // 0 .. 5 are the assembly's
  const double v8[8] = {e2, qnet, qabs_net, qabs_n, m_lin, m_d, m_after, bad};
  block_reduce<8, 4>(v8, red, part + 6 * gridDim.x + blockIdx.x, gridDim.x);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&w.count[b], 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = threadIdx.x >> 5; i < kP2Part; i += kP2Threads / 32) {
    const bool sum = i < 2 || (i >= 6 && i < 10);
    double t = 0.0;
    for (int q = threadIdx.x & 31; q < (int)gridDim.x; q += 32) {
      const double x = __ldcg(&part[i * gridDim.x + q]);
      t = sum ? t + x : fmax(t, x);
    }
    t = sum ? warp_sum(t) : warp_max(t);
    if ((threadIdx.x & 31) == 0) all[i] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    w.count[b] = 0;
    const double m_f = all[5], scale = fmax(fmax(all[2], all[3]), fmax(all[4], kQ));
    wg_poisson2d_info& o = info[b];
    const double lin = all[10] / fmax(m_f, kQ);
    o.converged = all[13] == 0.0 && isfinite(lin) && lin < 1e-8;
    o.linear_relres = lin;
    o.physical_relres_before = m_f / scale;
    o.physical_relres_after = all[12] / scale;
    o.physical_residual_before = m_f;
    o.residual_scale = scale;
    o.unmixed_step = all[11];
    o.iter_err = sqrt(all[6]);
    o.net_charge_per_length = -all[7];
    o.relative_charge_imbalance = fabs(all[7]) / fmax(kQ * fmax(all[8], all[9]), DBL_MIN);
    o.source_integral = all[0];
    o.target_integral = all[1];
  }
}

// M u on the full grid: the reference's operator with every row (free stencil rows, Dirichlet
// identity rows, phi(:,end) - phi(:,1) rows for the periodic duplicate).
__global__ void poisson2d_apply_kernel(P2Dev P, const double* __restrict__ u, double* __restrict__ y) {
  const size_t full = (size_t)P.nx * P.ny;
  const int b = blockIdx.y;
  u += b * full;
  y += b * full;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < full; k += (size_t)gridDim.x * blockDim.x) {
    const int ix = (int)(k % P.nx), iy = (int)(k / P.nx);
    if (P.periodic && iy == P.ny - 1) {
      y[k] = u[k] - u[ix];
      continue;
    }
    // unique-node stencil; a Y neighbour on the duplicate column reads column 0 (expand)
    const int ku = ix + iy * P.nx;
    if (P.fixed[ku]) {
      y[k] = u[k];
      continue;
    }
    double s = P.diag[ku] * u[k];
    if (ix > 0) s += P.cxm[ku] * u[k - 1];
    if (ix < P.nx - 1) s += P.cxp[ku] * u[k + 1];
    if (iy > 0) s += P.cym[ku] * u[k - P.nx];
    else if (P.periodic) s += P.cym[ku] * u[(size_t)(P.ny - 2) * P.nx + ix];
    if (iy < P.ny - 1) {
      const int jp = P.periodic && iy + 1 == P.ny - 1 ? 0 : iy + 1;
      s += P.cyp[ku] * u[(size_t)jp * P.nx + ix];
    }
    y[k] = s;
  }
}

template <typename T>
cudaError_t upload(T** d, const std::vector<T>& h) {
  cudaError_t e = cudaMalloc(d, std::max<size_t>(1, h.size()) * sizeof(T));
  if (e == cudaSuccess && !h.empty()) e = cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
  // the copy may return with its last part on the way, and the streams that read it do not wait for the default stream
  if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
  return e;
}

}  // namespace

struct wg_poisson2d {
  wg_poisson2d_desc d{};
  int nu = 0, NU = 0;
  P2Dev P{};
  cudaStream_t stream = nullptr;
  std::vector<void*> owned;
  double *src = nullptr, *phi0 = nullptr, *bc = nullptr, *phi = nullptr, *dens = nullptr, *work = nullptr;
  P2Work w{};
  wg_poisson2d_info* info = nullptr;
  bool projection = false;
  std::string msg;
};

namespace {

int fail(wg_poisson2d* h, int rc, const char* m) {
  if (h) h->msg = m;
  return rc;
}

template <typename T>
cudaError_t keep(wg_poisson2d* h, T** d, const std::vector<T>& v) {
  cudaError_t e = upload(d, v);
  if (e == cudaSuccess) h->owned.push_back((void*)*d);
  return e;
}

// Problems per group of launches: the grids' second dimension and the reduction's blocks (3 nx NU^2 doubles per
// problem) stay bounded for any batch.  A group of this size fills the chip at every level.
// With the chip full, operations count, and the reduction has three times those of a sweep over the columns: one warp per
// point sweeping would be faster from about 300 points of 32 rows, 450 of 24, 650 of 16 and 1,000 of 12 on (1,024 points
// of 361 columns: 60, 35, 16.7 and 10.5 ms against 141, 57, 21.1 and 10.9; 5.6 against 5.0 at 8 rows).  Not taken, since a
// point's bits would depend on the batch it is in.
constexpr int kP2Group = 1024;

cudaError_t launch_group(wg_poisson2d* h, int B, const double* src, int is_dg, const double* phi0, const double* bc,
                         int newton, double alpha, double* phi, double* dens, wg_poisson2d_info* info,
                         cudaStream_t st) {
  const double q_kt = kQ * kQ / (kKB * h->d.temp);
  const P2Dev& P = h->P;
  const P2Work& w = h->w;
  const dim3 nodes((unsigned)((P.nu * P.nx + kP2Threads - 1) / kP2Threads), B);
  int top = 1;
  while (P.nx / (2 * top) >= 1) top *= 2;
  poisson2d_assemble_kernel<<<nodes, kP2Threads, 0, st>>>(P, w, h->NU, src, is_dg, phi0, bc);
#define WG_P2_CASE(NU_)                                                                                          \
  case NU_:                                                                                                      \
    poisson2d_invert_kernel<NU_><<<dim3((unsigned)((P.nx + 1) / 2), B), ReduceShape<NU_, 2>::THREADS, 0, st>>>(  \
        P, w, newton, q_kt);                                                                                     \
    for (int s = 2; s <= top; s *= 2) {                                                                          \
      const dim3 grid((unsigned)(P.nx / s), B);                                                                  \
      if (s == 2)                                                                                                \
        poisson2d_reduce_kernel<NU_, true>                                                                       \
            <<<grid, ReduceShape<NU_, 3>::THREADS, 0, st>>>(P, w, newton, q_kt, s);                                 \
      else                                                                                                       \
        poisson2d_reduce_kernel<NU_, false>                                                                      \
            <<<grid, ReduceShape<NU_, 3>::THREADS, 0, st>>>(P, w, newton, q_kt, s);                                 \
    }                                                                                                            \
    if (top >= 8) poisson2d_back_kernel<NU_><<<dim3(1, B), kP2Threads, 0, st>>>(P, w, top, 8, 0);               \
    poisson2d_back_kernel<NU_>                                                                                   \
        <<<dim3((unsigned)((P.nx + 7) / 8), B), kP2Threads, 0, st>>>(P, w, std::min(top, 4), 1, 1);              \
    break;
  switch (h->NU) {
    WG_P2_CASE(4)
    WG_P2_CASE(8)
    WG_P2_CASE(12)
    WG_P2_CASE(16)
    WG_P2_CASE(24)
    WG_P2_CASE(32)
    default:
      return cudaErrorInvalidValue;
  }
#undef WG_P2_CASE
  poisson2d_finish_kernel<<<nodes, kP2Threads, 0, st>>>(P, w, h->NU, phi0, newton, q_kt, alpha, phi, dens, info);
  return cudaGetLastError();
}

cudaError_t launch_step(wg_poisson2d* h, const double* src, int is_dg, const double* phi0, const double* bc,
                        int newton, double alpha, double* phi, double* dens, cudaStream_t st) {
  const size_t full = (size_t)h->P.nx * h->P.ny, un = (size_t)h->P.nx * h->P.nu,
               ns = is_dg ? (size_t)h->P.ndx * h->P.ndy : full;
  cudaError_t e = cudaSuccess;
  for (int b = 0; b < h->d.batch && e == cudaSuccess; b += kP2Group)
    e = launch_group(h, std::min(kP2Group, h->d.batch - b), src + b * ns, is_dg, phi0 + b * full, bc + b * un, newton,
                     alpha, phi + b * full, dens + b * full, h->info + b, st);
  return e;
}

}  // namespace

extern "C" {

int wg_poisson2d_create(const wg_poisson2d_desc* d, const double* eps_r, const unsigned char* boundary,
                        const double* nd_m3, const double* na_m3, wg_poisson2d** out) {
  if (!d || !eps_r || !nd_m3 || !out) return WG_ERR_ARG;
  *out = nullptr;
  const int nx = d->nx, ny = d->ny, B = d->batch;
  if (nx < 2 || ny < 1 || B < 1 || !(d->dx_nm > 0) || !(d->dy_nm > 0) || !std::isfinite(d->dx_nm) ||
      !std::isfinite(d->dy_nm) || !(d->temp > 0))
    return WG_ERR_ARG;
  const int periodic = d->periodic_y ? 1 : 0;
  if (periodic && ny < 3) return WG_ERR_ARG;                       // RTD:PoissonPeriodicMaterial
  const int nu = ny - periodic;
  if (nu > 32) return WG_ERR_ARG;                                   // the widest blocks of the reduction
  const size_t full = (size_t)nx * ny;
  double emax = 0.0;
  for (size_t k = 0; k < full; ++k) {
    if (!(eps_r[k] > 0) || !std::isfinite(eps_r[k])) return WG_ERR_ARG;
    emax = std::max(emax, eps_r[k]);
    if (!(nd_m3[k] >= 0) || !std::isfinite(nd_m3[k]) || (na_m3 && (!(na_m3[k] >= 0) || !std::isfinite(na_m3[k]))))
      return WG_ERR_ARG;
  }
  auto at = [&](const double* a, int ix, int iy) { return a[(size_t)iy * nx + ix]; };
  if (periodic)
    for (int ix = 0; ix < nx; ++ix)
      if (std::fabs(at(eps_r, ix, ny - 1) - at(eps_r, ix, 0)) > 1e-12 * emax) return WG_ERR_ARG;
  std::vector<unsigned char> fixedf(full, 0);
  if (boundary) {
    for (size_t k = 0; k < full; ++k) fixedf[k] = boundary[k] ? 1 : 0;
  } else if (!d->neumann_x) {
    for (int iy = 0; iy < ny; ++iy) fixedf[(size_t)iy * nx] = fixedf[(size_t)iy * nx + nx - 1] = 1;
  }
  bool any = false;
  for (unsigned char f : fixedf) any = any || f;
  if (d->neumann_x && any) return WG_ERR_ARG;                       // RTD:PoissonBoundaryConflict
  if (!d->neumann_x && !any) return WG_ERR_ARG;                     // Dirichlet needs a fixed node
  if (periodic)
    for (int ix = 0; ix < nx; ++ix)
      if (fixedf[(size_t)(ny - 1) * nx + ix] != fixedf[ix]) return WG_ERR_ARG;   // RTD:PoissonPeriodicBoundary

  // the stencil of the unique rows (eval_Poisson2D_rtd.m:118-185)
  const int nun = nu * nx;
  std::vector<unsigned char> fx(nun);
  std::vector<double> cxm(nun, 0.0), cxp(nun, 0.0), cym(nun, 0.0), cyp(nun, 0.0), dg(nun, 0.0), net(nun);
  const double cx = kEps0 * 1e18 / (d->dx_nm * d->dx_nm), cy = kEps0 * 1e18 / (d->dy_nm * d->dy_nm);
  auto hm = [](double a, double b) { return 2 * a * b / (a + b); };
  for (int iy = 0; iy < nu; ++iy)
    for (int ix = 0; ix < nx; ++ix) {
      const int k = ix + iy * nx;
      fx[k] = fixedf[(size_t)iy * nx + ix];
      net[k] = at(nd_m3, ix, iy) - (na_m3 ? at(na_m3, ix, iy) : 0.0);
      if (fx[k]) continue;
      const double e0 = at(eps_r, ix, iy);
      double diag = 0.0;
      if (ix > 0) {
        double c = cx * hm(e0, at(eps_r, ix - 1, iy));
        if (ix == nx - 1) c *= 2;
        cxm[k] = c;
        diag -= c;
      }
      if (ix < nx - 1) {
        double c = cx * hm(e0, at(eps_r, ix + 1, iy));
        if (ix == 0) c *= 2;
        cxp[k] = c;
        diag -= c;
      }
      if (iy > 0 || periodic) {
        const int jm = iy > 0 ? iy - 1 : ny - 2;
        double c = cy * hm(e0, at(eps_r, ix, jm));
        if (!periodic && iy == ny - 1) c *= 2;
        cym[k] = c;
        diag -= c;
      }
      if (iy < ny - 1) {
        int jp = iy + 1;
        if (periodic && jp == ny - 1) jp = 0;
        double c = cy * hm(e0, at(eps_r, ix, jp));
        if (!periodic && iy == 0) c *= 2;
        cyp[k] = c;
        diag -= c;
      }
      dg[k] = diag;
    }
  // control-volume widths of the charge diagnostics (solve_Poisson2D_rtd.m:115-118)
  std::vector<double> vx(nx, d->dx_nm * 1e-9), vy(nu, d->dy_nm * 1e-9);
  vx[0] /= 2;
  vx[nx - 1] /= 2;
  if (!periodic && nu > 1) {
    vy[0] /= 2;
    vy[nu - 1] /= 2;
  }
  wg_poisson2d* h = new wg_poisson2d;
  h->d = *d;
  h->d.periodic_y = periodic;
  h->nu = nu;
  h->NU = nu <= 4 ? 4 : nu <= 8 ? 8 : nu <= 12 ? 12 : nu <= 16 ? 16 : nu <= 24 ? 24 : 32;
  P2Dev& P = h->P;
  P.nx = nx;
  P.ny = ny;
  P.nu = nu;
  P.periodic = periodic;
  P.batch = B;
  cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  unsigned char* dfx = nullptr;
  double *dcxm = nullptr, *dcxp = nullptr, *dcym = nullptr, *dcyp = nullptr, *ddg = nullptr, *dnet = nullptr,
         *dvx = nullptr, *dvy = nullptr;
  if (e == cudaSuccess) e = keep(h, &dfx, fx);
  if (e == cudaSuccess) e = keep(h, &dcxm, cxm);
  if (e == cudaSuccess) e = keep(h, &dcxp, cxp);
  if (e == cudaSuccess) e = keep(h, &dcym, cym);
  if (e == cudaSuccess) e = keep(h, &dcyp, cyp);
  if (e == cudaSuccess) e = keep(h, &ddg, dg);
  if (e == cudaSuccess) e = keep(h, &dnet, net);
  if (e == cudaSuccess) e = keep(h, &dvx, vx);
  if (e == cudaSuccess) e = keep(h, &dvy, vy);
  P.fixed = dfx;
  P.cxm = dcxm;
  P.cxp = dcxp;
  P.cym = dcym;
  P.cyp = dcyp;
  P.diag = ddg;
  P.net = dnet;
  P.vx = dvx;
  P.vy = dvy;
  const size_t sz = (size_t)B * full * sizeof(double);
  if (e == cudaSuccess) e = cudaMalloc(&h->src, sz);
  if (e == cudaSuccess) e = cudaMalloc(&h->phi0, sz);
  if (e == cudaSuccess) e = cudaMalloc(&h->bc, (size_t)B * nun * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&h->phi, sz);
  if (e == cudaSuccess) e = cudaMalloc(&h->dens, sz);
  {
    const size_t G = std::min(B, kP2Group), bb = (size_t)h->NU * h->NU, half = G * (nx / 2) * bb,
                 even = G * ((nx + 1) / 2) * bb, col = G * nx * h->NU, un = G * nun,
                 part = G * kP2Part * ((nun + kP2Threads - 1) / kP2Threads);
    double** const ptr[] = {&h->w.n, &h->w.v, &h->w.F, &h->w.r, &h->w.y, &h->w.d,    &h->w.D,
                            &h->w.L, &h->w.U, &h->w.XL, &h->w.XU, &h->w.Dinv, &h->w.part};
    const size_t len[] = {un, un, un, col, col, col, half, half, half, half, half, even, part};
    size_t total = 0;
    for (size_t l : len) total += l;
    if (e == cudaSuccess) e = cudaMalloc(&h->work, total * sizeof(double));
    size_t at0 = 0;
    for (int i = 0; i < 13; ++i) {
      *ptr[i] = h->work + at0;
      at0 += len[i];
    }
    if (e == cudaSuccess) e = cudaMalloc(&h->w.count, G * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(h->w.count, 0, G * sizeof(int));
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
  }
  if (e == cudaSuccess) e = cudaMalloc(&h->info, (size_t)B * sizeof(wg_poisson2d_info));
  if (e != cudaSuccess) {
    wg_poisson2d_destroy(h);
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? WG_ERR_OOM : WG_ERR_CUDA;
  }
  *out = h;
  return WG_OK;
}

int wg_poisson2d_destroy(wg_poisson2d* h) {
  if (!h) return WG_OK;
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (void* p : h->owned) cudaFree(p);
  for (void* p : {(void*)h->src, (void*)h->phi0, (void*)h->bc, (void*)h->phi, (void*)h->dens, (void*)h->work,
                  (void*)h->w.count, (void*)h->info})
    if (p) cudaFree(p);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return WG_OK;
}

const char* wg_poisson2d_last_error(const wg_poisson2d* h) { return h ? h->msg.c_str() : "null handle"; }

int wg_poisson2d_set_projection(wg_poisson2d* h, int ndof_x, const int* tx_rp, const int* tx_col, const double* tx_val,
                                int ndof_y, const int* ty_rp, const int* ty_col, const double* ty_val,
                                const double* wx, const double* wy, const double* src_x, const double* src_y) {
  if (!h || ndof_x < 1 || ndof_y < 1 || !tx_rp || !tx_col || !tx_val || !ty_rp || !ty_col || !ty_val || !wx || !wy ||
      !src_x || !src_y)
    return WG_ERR_ARG;
  const int nx = h->d.nx, nu = h->nu;
  if (tx_rp[0] != 0 || ty_rp[0] != 0) return fail(h, WG_ERR_ARG, "CSR row pointers must start at 0");
  for (int i = 0; i < nx; ++i)
    if (tx_rp[i + 1] < tx_rp[i]) return fail(h, WG_ERR_ARG, "Tx row pointers must not decrease");
  for (int i = 0; i < nu; ++i)
    if (ty_rp[i + 1] < ty_rp[i]) return fail(h, WG_ERR_ARG, "Ty row pointers must not decrease");
  for (int p = 0; p < tx_rp[nx]; ++p)
    if (tx_col[p] < 0 || tx_col[p] >= ndof_x) return fail(h, WG_ERR_ARG, "Tx column out of range");
  for (int p = 0; p < ty_rp[nu]; ++p)
    if (ty_col[p] < 0 || ty_col[p] >= ndof_y) return fail(h, WG_ERR_ARG, "Ty column out of range");
  for (int i = 0; i < nx; ++i)
    if (!(wx[i] > 0)) return fail(h, WG_ERR_ARG, "dual-volume widths must be positive");
  for (int i = 0; i < nu; ++i)
    if (!(wy[i] > 0)) return fail(h, WG_ERR_ARG, "dual-volume widths must be positive");
  std::vector<int> vtr(tx_rp, tx_rp + nx + 1), vtc(tx_col, tx_col + tx_rp[nx]), vyr(ty_rp, ty_rp + nu + 1),
      vyc(ty_col, ty_col + ty_rp[nu]);
  std::vector<double> vtv(tx_val, tx_val + tx_rp[nx]), vyv(ty_val, ty_val + ty_rp[nu]), vwx(wx, wx + nx),
      vwy(wy, wy + nu), vsx(src_x, src_x + ndof_x), vsy(src_y, src_y + ndof_y);
  P2Dev& P = h->P;
  int *a = nullptr, *b = nullptr, *c = nullptr, *dd = nullptr;
  double *e1 = nullptr, *e2 = nullptr, *e3 = nullptr, *e4 = nullptr, *e5 = nullptr, *e6 = nullptr;
  cudaError_t e = keep(h, &a, vtr);
  if (e == cudaSuccess) e = keep(h, &b, vtc);
  if (e == cudaSuccess) e = keep(h, &c, vyr);
  if (e == cudaSuccess) e = keep(h, &dd, vyc);
  if (e == cudaSuccess) e = keep(h, &e1, vtv);
  if (e == cudaSuccess) e = keep(h, &e2, vyv);
  if (e == cudaSuccess) e = keep(h, &e3, vwx);
  if (e == cudaSuccess) e = keep(h, &e4, vwy);
  if (e == cudaSuccess) e = keep(h, &e5, vsx);
  if (e == cudaSuccess) e = keep(h, &e6, vsy);
  if (e != cudaSuccess) return fail(h, WG_ERR_CUDA, cudaGetErrorString(e));
  if ((size_t)ndof_x * ndof_y > (size_t)h->d.nx * h->d.ny) {
    // the source buffer holds nDG for the host entry points
    cudaFree(h->src);
    h->src = nullptr;
    e = cudaMalloc(&h->src, (size_t)h->d.batch * ndof_x * ndof_y * sizeof(double));
    if (e != cudaSuccess) return fail(h, WG_ERR_OOM, "source buffer");
  }
  P.ndx = ndof_x;
  P.ndy = ndof_y;
  P.tx_rp = a;
  P.tx_col = b;
  P.ty_rp = c;
  P.ty_col = dd;
  P.tx_val = e1;
  P.ty_val = e2;
  P.wx = e3;
  P.wy = e4;
  P.srcx = e5;
  P.srcy = e6;
  h->projection = true;
  return WG_OK;
}

int wg_poisson2d_apply(wg_poisson2d* h, const double* phi, double* out) {
  if (!h || !phi || !out) return WG_ERR_ARG;
  const size_t sz = (size_t)h->d.batch * h->d.nx * h->d.ny * sizeof(double);
  cudaError_t e = cudaMemcpyAsync(h->phi0, phi, sz, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess) {
    dim3 grid((unsigned)std::min<size_t>(1024, ((size_t)h->d.nx * h->d.ny + 255) / 256), h->d.batch);
    poisson2d_apply_kernel<<<grid, 256, 0, h->stream>>>(h->P, h->phi0, h->phi);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, h->phi, sz, cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  return e == cudaSuccess ? WG_OK : fail(h, WG_ERR_CUDA, cudaGetErrorString(e));
}

int wg_poisson2d_contacts(wg_poisson2d* h, const double* bias, const double* vbc, double* bc_out) {
  // solve_Poisson2D_rtd.m:50-52: bc(end,:) = bias unless mat.Vbc gives the contact potential
  if (!h || !bc_out || (!bias && !vbc)) return WG_ERR_ARG;
  const int nx = h->d.nx, nu = h->nu, B = h->d.batch;
  for (int b = 0; b < B; ++b)
    for (int iy = 0; iy < nu; ++iy)
      for (int ix = 0; ix < nx; ++ix) {
        const size_t k = (size_t)b * nu * nx + (size_t)iy * nx + ix;
        bc_out[k] = vbc ? vbc[(size_t)b * nx * h->d.ny + (size_t)iy * nx + ix] : (ix == nx - 1 ? bias[b] : 0.0);
      }
  return WG_OK;
}

int wg_poisson2d_solve_device(wg_poisson2d* h, const double* src, int src_is_dg, const double* phi0,
                              const double* bc, int newton, double alpha, double* phi, double* density, void* stream) {
  if (!h || !src || !phi0 || !bc || !phi || !density || !(alpha > 0 && alpha <= 1)) return WG_ERR_ARG;
  if (src_is_dg && !h->projection) return fail(h, WG_ERR_ARG, "wg_poisson2d_set_projection first");
  if (!newton && h->d.neumann_x) return fail(h, WG_ERR_ARG, "RTD:NeumannNeedsNewton");
  cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
  const cudaError_t e = launch_step(h, src, src_is_dg, phi0, bc, newton, alpha, phi, density, st);
  return e == cudaSuccess ? WG_OK : fail(h, WG_ERR_CUDA, cudaGetErrorString(e));
}

int wg_poisson2d_info_get(wg_poisson2d* h, void* stream, wg_poisson2d_info* info) {
  if (!h || !info) return WG_ERR_ARG;
  cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
  cudaError_t e = cudaMemcpyAsync(info, h->info, (size_t)h->d.batch * sizeof(wg_poisson2d_info),
                                  cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? WG_OK : fail(h, WG_ERR_CUDA, cudaGetErrorString(e));
}

int wg_poisson2d_solve(wg_poisson2d* h, const double* src, int src_is_dg, const double* phi0, const double* bias,
                       const double* vbc, int newton, double alpha, double* phi, double* density,
                       wg_poisson2d_info* info) {
  if (!h || !src || !phi0 || !phi || !density || !info || (!bias && !vbc)) return WG_ERR_ARG;
  const int nx = h->d.nx, ny = h->d.ny, B = h->d.batch;
  const size_t full = (size_t)nx * ny;
  if (src_is_dg && !h->projection) return fail(h, WG_ERR_ARG, "wg_poisson2d_set_projection first");
  if (h->d.neumann_x && !newton) return fail(h, WG_ERR_ARG, "RTD:NeumannNeedsNewton");
  if (h->d.neumann_x && vbc) return fail(h, WG_ERR_ARG, "RTD:PoissonBoundaryConflict");
  const size_t nsrc = src_is_dg ? (size_t)h->P.ndx * h->P.ndy : full;
  for (size_t k = 0; k < (size_t)B * nsrc; ++k)
    if (!std::isfinite(src[k])) return fail(h, WG_ERR_ARG, "density must be finite");
  for (size_t k = 0; k < (size_t)B * full; ++k)
    if (!std::isfinite(phi0[k])) return fail(h, WG_ERR_ARG, "phi0 must be finite");
  if (!src_is_dg && h->d.neumann_x) {
    // solve_Poisson2D_rtd.m:97-100: Newton screening needs a non-negative, non-zero density
    for (int b = 0; b < B; ++b) {
      bool pos = false;
      for (size_t k = 0; k < full; ++k) {
        if (src[b * full + k] < 0) return fail(h, WG_ERR_ARG, "RTD:NeumannDensityResponse");
        pos = pos || src[b * full + k] > 0;
      }
      if (!pos) return fail(h, WG_ERR_ARG, "RTD:NeumannDensityResponse");
    }
  }
  if (h->d.periodic_y) {
    // solve_Poisson2D_rtd.m:53-57 and 133-137: the included Y endpoints must agree
    auto periodic_ok = [&](const double* a) {
      for (int b = 0; b < B; ++b) {
        double mx = 1.0;
        for (size_t k = 0; k < full; ++k) mx = std::max(mx, std::fabs(a[b * full + k]));
        for (int ix = 0; ix < nx; ++ix)
          if (std::fabs(a[b * full + ix] - a[b * full + (size_t)(ny - 1) * nx + ix]) > 1e-10 * mx) return false;
      }
      return true;
    };
    if ((!src_is_dg && !periodic_ok(src)) || !periodic_ok(phi0) || (vbc && !periodic_ok(vbc)))
      return fail(h, WG_ERR_ARG, "RTD:NonperiodicPoissonData");
  }
  std::vector<double> bc((size_t)B * h->nu * nx);
  int rc = wg_poisson2d_contacts(h, bias, vbc, bc.data());
  if (rc != WG_OK) return rc;
  cudaError_t e = cudaMemcpyAsync(h->src, src, (size_t)B * nsrc * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->phi0, phi0, (size_t)B * full * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->bc, bc.data(), bc.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess) e = launch_step(h, h->src, src_is_dg, h->phi0, h->bc, newton, alpha, h->phi, h->dens, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(phi, h->phi, (size_t)B * full * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(density, h->dens, (size_t)B * full * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  if (e != cudaSuccess) return fail(h, WG_ERR_CUDA, cudaGetErrorString(e));
  rc = wg_poisson2d_info_get(h, h->stream, info);
  if (rc != WG_OK) return rc;
  return WG_OK;
}

int wg_poisson2d_buffers(wg_poisson2d* h, double** src, double** phi0, double** bc, double** phi, double** density) {
  if (!h) return WG_ERR_ARG;
  if (src) *src = h->src;
  if (phi0) *phi0 = h->phi0;
  if (bc) *bc = h->bc;
  if (phi) *phi = h->phi;
  if (density) *density = h->dens;
  return WG_OK;
}

}  // extern "C"
