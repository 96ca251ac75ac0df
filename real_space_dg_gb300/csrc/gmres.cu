// Batched restarted GMRES(m) with right preconditioning (sm_103a).
//
// Semantics of the reference's Krylov wrapper (DG_code/solve_transport_DG_full2D.m):
//  - right preconditioning: Krylov space of A M^-1, x = x0 + M^-1 V y (:462-484)
//  - warm start as a correction about rho0 with the absolute target tol*|b| (:474)
//  - an independent true-residual check that downgrades a converged flag (:314-320)
// Arnoldi uses classical Gram-Schmidt applied twice (CGS2) with block reductions
// and warp shuffles; Givens rotations and the Hessenberg back substitution run on
// the device, one warp per problem.  Every problem of a batch has its own basis,
// Hessenberg matrix and convergence state; a converged problem freezes.
//
// Two drivers share the Arnoldi step, templated on the basis vector type:
//  - gmres_solve_fp64:  FP64 basis and operator (the drop-in plain form);
//  - gmres_solve_mixed: FP64 iterative refinement.  The outer residual
//    r = b - A x is FP64; each correction solves A d = r/|r| with one GMRES cycle
//    whose basis is stored in FP16 (FP32 with inner_basis_fp32), with FP32
//    arithmetic, and whose operator runs the BF16 tensor-core transforms and the
//    FP32 flux / preconditioner.  Inner products and norms are combined in FP64
//    (see AccF32), Givens rotations and the Hessenberg solve are FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <type_traits>

#include "krylov.cuh"
#include "problem.h"

namespace wg {

namespace {

__device__ __forceinline__ double2 ld2(const double2& v) { return v; }
__device__ __forceinline__ double2 ld2(const float2& v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ void st2(double2& d, double2 v) { d = v; }
__device__ __forceinline__ void st2(float2& d, double2 v) { d = make_float2((float)v.x, (float)v.y); }

// Inner-product accumulators.  FP64 vectors accumulate in FP64.  FP32 basis
// vectors (mixed form) multiply and add in FP32 within a thread (at most 8
// complex terms) and across the warp (a 5-level tree), then in FP64 across warps,
// blocks and chunks.  The error, a few 1e-7 of sum |a_i b_i|, matches the rounding
// of the FP32 basis itself; the inner GMRES it serves targets 1e-3.  (Error-free
// FP32 transformations per element measured at a third of the HBM rate, and
// double-float merges per warp level made the kernels issue-bound.)
struct Acc64 {
  double2 v = make_double2(0.0, 0.0);
  __device__ __forceinline__ void add_cdot(const double2& a, const double2& x) {  // += conj(a) x
    v.x = fma(a.x, x.x, fma(a.y, x.y, v.x));
    v.y = fma(a.x, x.y, fma(-a.y, x.x, v.y));
  }
  __device__ __forceinline__ void add_norm(const double2& a) { v.x = fma(a.x, a.x, fma(a.y, a.y, v.x)); }
  __device__ __forceinline__ void warp_reduce() {
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
  }
  __device__ __forceinline__ double2 get() const { return v; }
  // block-level staging: one slot of 4 doubles per warp
  __device__ __forceinline__ void stage(double* slot) const { slot[0] = v.x; slot[1] = v.y; }
  __device__ __forceinline__ static double2 combine(const double* slots, int n) {
    double2 r = make_double2(0, 0);
    for (int q = 0; q < n; ++q) { r.x += slots[4 * q]; r.y += slots[4 * q + 1]; }
    return r;
  }
};

struct AccF32 {
  float re = 0.f, im = 0.f;
  __device__ __forceinline__ void add_cdot(const float2& a, const float2& x) {
    re = fmaf(a.x, x.x, fmaf(a.y, x.y, re));
    im = fmaf(a.x, x.y, fmaf(-a.y, x.x, im));
  }
  __device__ __forceinline__ void add_norm(const float2& a) { re = fmaf(a.x, a.x, fmaf(a.y, a.y, re)); }
  __device__ __forceinline__ void warp_reduce() {
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
  }
  __device__ __forceinline__ void stage(double* slot) const {
    float* f = reinterpret_cast<float*>(slot);
    f[0] = re;
    f[1] = im;
  }
  __device__ __forceinline__ static double2 combine(const double* slots, int n) {
    double2 r = make_double2(0, 0);
    for (int q = 0; q < n; ++q) {
      const float* f = reinterpret_cast<const float*>(slots + 4 * q);
      r.x += (double)f[0];
      r.y += (double)f[1];
    }
    return r;
  }
};

template <typename T> struct AccFor;
template <> struct AccFor<double2> { using type = Acc64; };
template <> struct AccFor<float2> { using type = AccF32; };

// hcol[b][i] = sum_c partial[b][i][c] (FP64); H[b][k][i] = (first; diag added at i = k) or += hcol.  One block.
__device__ void dot_reduce_block(const double2* __restrict__ partial, double2* __restrict__ hcol,
                                 float2* __restrict__ hcol32, double2* __restrict__ H, int b, int nv, int k,
                                 int pstride, int m, int nchunk, int first, double diag) {
  // warp w takes the coefficients w, w + nw, w + 2 nw, w + 3 nw together, so that the loads
  // of four partial rows are in flight at once (this tail runs after the grid's last block)
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i0 = w; i0 < nv; i0 += U * nw) {
    double2 acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = make_double2(0, 0);
#pragma unroll 2
    for (int c = lane; c < nchunk; c += 32) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * nw;
        if (i < nv) {
          const double2 t = __ldcg(&partial[((long long)b * pstride + i) * nchunk + c]);
          acc[u].x += t.x;
          acc[u].y += t.y;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * nw;
      if (i >= nv) continue;   // warp-uniform
      acc[u].x = warp_sum(acc[u].x);
      acc[u].y = warp_sum(acc[u].y);
      if (lane == 0) {
        hcol[b * pstride + i] = acc[u];
        if (hcol32) hcol32[b * pstride + i] = make_float2((float)acc[u].x, (float)acc[u].y);
        double2* h = H + (long long)b * pstride * m + (long long)k * pstride + i;
        if (first) *h = make_double2(acc[u].x + (i == k ? diag : 0.0), acc[u].y);
        else { h->x += acc[u].x; h->y += acc[u].y; }
      }
    }
  }
}

// Arguments of the per-problem tail work done by the last block of a launch.
struct KrylovTail {
  int* md_count;       // [B] tickets of the multi-dot
  int* gs_count;       // [B] tickets of the update
  double2* partial;    // multi-dot partials
  double2* hcol;       // FP64 coefficients
  float2* hcol32;      // FP32 copy (mixed form) or null
  double2* H;
  double2 *cs, *sn, *g;
  int* active;
  int* kused;
  int* reorth;
  const double* target;
  double* nrm;
  double* inv64;
  float* inv32;
  double eta2;         // DGKS threshold squared
  double diag;         // added to H[k][k]: 1 when w is A M^-1 v_k - v_k (flux_is_inverted)
  int k, pstride, m, first;
};

// Sums over a warp of 8 values per lane: 9 shuffles and additions instead of 40 (each step exchanges half of
// the values still held).  Lane l returns the sum of v[l >> 2].
template <typename R>
__device__ __forceinline__ R warp_sum8(R (&v)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4; h >= 1; h /= 2) {
    const bool up = lane & (4 * h);
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const R give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * h);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// Multi-dot: partial[b][i][c] = sum over chunk c of conj(V_i) . w for every i < nv; the last block of problem b
// reduces the partials into the Hessenberg column.  The warps drop their sums of four vectors (real and
// imaginary parts: 8 values) in shared memory and the block adds them at the end.
//
// FP32 vectors, basis of VB (FP16 or FP32): one block per (`quads` groups of four elements, problem; dot_quads); 2,048
// elements of w at a time stay in registers, two basis vectors are loaded (16 bytes per load) while two are summed.
// Bound by HBM; with few vectors by the fixed latencies of a block (w, the fence and the ticket), which every further
// wave of blocks pays again.  16 problems of 245,760 unknowns, 21 vectors: 73 us, 5.0 TB/s (82 us with 20 vectors where a
// block took one chunk of 2,048 elements and reduced it vector by vector).  Tried and slower: the copies through a
// shared-memory ring, and this kernel and the update in one launch by problem so that the basis stays in the L2 (150 us
// against 141 us for both).
template <typename VB>
__global__ void __launch_bounds__(256, 3) multidot32_kernel(const VB* __restrict__ V, const float2* __restrict__ w,
                                                            double2* __restrict__ partial,
                                                            const int* __restrict__ active, long long N, int nv,
                                                            int mp1, int pstride, int nchunk, int quads,
                                                            KrylovTail tl) {
  extern __shared__ double red32[];  // [nv rounded up to 4][2][8 warps]
  const int b = blockIdx.y, c = blockIdx.x;
  if (!active[b]) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long lo = (long long)c * quads, hi = min(N / 4, lo + quads);
  const VB* v = V + (long long)b * mp1 * N;
  for (long long base = lo; base < hi; base += 512) {
    const long long n0 = base + threadIdx.x, n1 = n0 + 256;
    const bool in0 = n0 < hi, in1 = n1 < hi;
    Quad<float2> w0, w1;
    w0.zero();
    w1.zero();
    if (in0) w0.load(w + (long long)b * N, n0);
    if (in1) w1.load(w + (long long)b * N, n1);
    // two vectors are in flight while two are summed
    Quad<VB> a0[4], a1[4];
    auto load2 = [&](int i, int u0) {
#pragma unroll
      for (int u = u0; u < u0 + 2; ++u) {
        a0[u].zero();
        a1[u].zero();
        if (i + u < nv && in0) a0[u].load(v + (long long)(i + u) * N, n0);
        if (i + u < nv && in1) a1[u].load(v + (long long)(i + u) * N, n1);
      }
    };
    load2(0, 0);
    for (int i = 0; i < nv; i += 4) {
      float s[8];
      load2(i, 2);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        AccF32 t;
#pragma unroll
        for (int q = 0; q < 4; ++q) t.add_cdot(a0[u].get(q), w0.get(q));
#pragma unroll
        for (int q = 0; q < 4; ++q) t.add_cdot(a1[u].get(q), w1.get(q));
        s[2 * u] = t.re;
        s[2 * u + 1] = t.im;
        if (u == 1) load2(i + 4, 0);
      }
      const float r = warp_sum8(s);
      if ((lane & 3) == 0) {   // always the same thread's slot
        double* d = red32 + (2 * i + (lane >> 2)) * 8 + warp;
        *d = base == lo ? (double)r : *d + (double)r;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    double2 r = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      r.x += red32[16 * i + q];
      r.y += red32[16 * i + 8 + q];
    }
    partial[((long long)b * pstride + i) * nchunk + c] = r;
  }
  if (!last_block_of_problem(tl.md_count, b)) return;
  dot_reduce_block(partial, tl.hcol, tl.hcol32, tl.H, b, nv, tl.k, pstride, tl.m, nchunk, tl.first, tl.diag);
  if (threadIdx.x == 0) tl.md_count[b] = 0;
}

// FP64: one block per (256 E elements, problem, four vectors).  Bound by the FP64 pipe (4 FMAs per element and
// vector), so the vectors are split over blocks: the 608 pipe quarters fill evenly at any nv, and a small
// problem is not one block that takes its vectors one after another.  E (Problem::md_e) is the largest of
// 8, 4, 2, 1 that still gives a few blocks per SM.
// 2 problems of 245,760 unknowns, 25 vectors: 214 -> 111 us against whole problems per block and a multiply, FMA
// and add per product (0.81 TFLOP/s); 1,152 unknowns: 109 -> 13 us.
template <int E>
__global__ void __launch_bounds__(256) multidot64_kernel(const double2* __restrict__ V, const double2* __restrict__ w,
                                                         double2* __restrict__ partial,
                                                         const int* __restrict__ active, long long N, int nv, int mp1,
                                                         int pstride, int nchunk, KrylovTail tl) {
  __shared__ double red[8][8];
  const int b = blockIdx.y, c = blockIdx.x, i0 = 4 * blockIdx.z;
  if (!active[b]) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)c * 256 * E + threadIdx.x;
  const double2* wb = w + (long long)b * N;
  const double2* v = V + ((long long)b * mp1 + i0) * N;
  Acc64 acc[4];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const long long n = base + (long long)j * 256;
    if (n < N) {
      const double2 x = __ldg(wb + n);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < nv) acc[u].add_cdot(__ldg(v + (long long)u * N + n), x);
    }
  }
  double s[8];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    s[2 * u] = acc[u].v.x;
    s[2 * u + 1] = acc[u].v.y;
  }
  const double r = warp_sum8(s);
  if ((lane & 3) == 0) red[lane >> 2][warp] = r;
  __syncthreads();
  if (threadIdx.x < 4 && i0 + (int)threadIdx.x < nv) {
    double2 t = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      t.x += red[2 * threadIdx.x][q];
      t.y += red[2 * threadIdx.x + 1][q];
    }
    partial[((long long)b * pstride + i0 + threadIdx.x) * nchunk + c] = t;
  }
  if (!last_block_of_problem(tl.md_count, b)) return;
  dot_reduce_block(partial, tl.hcol, tl.hcol32, tl.H, b, nv, tl.k, pstride, tl.m, nchunk, tl.first, tl.diag);
  if (threadIdx.x == 0) tl.md_count[b] = 0;
}

// What follows the update w -= sum_i V_i hcol_i: nrm_partial[b][block] = sum |w|^2 (a: the thread's share), and
// the last block of problem b finishes the step.  MODE 1 runs the DGKS test (reorth[b]) and, when no second
// pass is needed, MODE 2's work: |w|, H[k+1][k], inverse norm, Givens step.
template <int MODE, typename Acc>
__device__ void update_tail(Acc& a, const int b, double* __restrict__ nrm_partial, int nv, int pstride, int nblk,
                            const KrylovTail& tl) {
  __shared__ double wsum[8 * 4];
  a.warp_reduce();
  if ((threadIdx.x & 31) == 0) a.stage(wsum + (threadIdx.x >> 5) * 4);
  __syncthreads();
  if (threadIdx.x == 0)
    nrm_partial[(long long)b * nblk + blockIdx.x] = Acc::combine(wsum, blockDim.x >> 5).x;
  if (!last_block_of_problem(tl.gs_count, b)) return;
  // the whole last block adds the partial norms (independent loads), warp 0 finishes the step
  double w2p = 0;
#pragma unroll 4
  for (int c = threadIdx.x; c < nblk; c += blockDim.x) w2p += __ldcg(&nrm_partial[(long long)b * nblk + c]);
  const double w2b = block_sum1(w2p);
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const double w2 = __shfl_sync(0xffffffffu, w2b, 0);
    bool finish = true;
    if (MODE == 1) {
      double h2 = 0;
      for (int i = lane; i < nv; i += 32) {
        const double2 h = tl.hcol[(long long)b * pstride + i];
        h2 += h.x * h.x + h.y * h.y;
      }
      h2 = warp_sum(h2);
      const int re = w2 < tl.eta2 * (w2 + h2) ? 1 : 0;
      if (lane == 0) tl.reorth[b] = re;
      finish = !re;
    }
    if (finish) {
      const double inv = w2 > 0 ? rsqrt(w2) : 0.0;
      const double v = w2 > 0 ? w2 * inv : w2;   // NaN passes on
      if (lane == 0) {
        tl.nrm[b] = v;
        if (tl.inv64) tl.inv64[b] = inv;
        if (tl.inv32) tl.inv32[b] = (float)inv;
      }
      givens_warp(tl.H, tl.cs, tl.sn, tl.g, tl.active, tl.kused, tl.target, b, tl.k, pstride, tl.m, v);
    }
  }
  if (threadIdx.x == 0) tl.gs_count[b] = 0;
}

// w -= sum_i V_i hcol_i, FP32 vectors: 128 threads of four consecutive complex values, the loads of eight
// basis vectors in flight per thread (16 bytes each of an FP16 basis), the next four before the last four are used.
// Bound by HBM.  The problems in the reverse of the multi-dot's order, so that the basis vectors that one of the two
// reads last are the first of the other while they are in the L2.  16 problems of 245,760 unknowns, 21 vectors: 70 us,
// 5.5 TB/s (105 us with 20 vectors at 512 elements a block).
constexpr int kUp32Threads = 128;
template <int MODE, typename VB>
__global__ void __launch_bounds__(kUp32Threads, 8) gs_update32_kernel(const VB* __restrict__ V,
                                                                      float2* __restrict__ w,
                                                                      const float2* __restrict__ hcol,
                                                                      const int* __restrict__ mask,
                                                                      double* __restrict__ nrm_partial, long long N,
                                                                      int nv, int mp1, int pstride, int nblk,
                                                                      int quads, KrylovTail tl) {
  const int b = gridDim.y - 1 - blockIdx.y;
  if (!mask[b]) return;
  __shared__ float2 hs[kMaxRestart + 8];
  for (int i = threadIdx.x; i < ((nv + 7) & ~7); i += kUp32Threads)
    hs[i] = i < nv ? hcol[b * pstride + i] : make_float2(0.f, 0.f);
  const long long lo = (long long)blockIdx.x * quads, hi = min(N / 4, lo + quads);
  const VB* v = V + (long long)b * mp1 * N;
  __syncthreads();
  constexpr int U = sizeof(VB) == 4 ? 8 : 4;
  double nrm2 = 0.0;   // sums of four values in FP32
  for (long long n4 = lo + threadIdx.x; n4 < hi; n4 += kUp32Threads) {
    float4* wp = reinterpret_cast<float4*>(w + (long long)b * N) + 2 * n4;
    const float4 x0 = wp[0], x1 = wp[1];
    float2 acc[4] = {make_float2(x0.x, x0.y), make_float2(x0.z, x0.w), make_float2(x1.x, x1.y),
                     make_float2(x1.z, x1.w)};
    Quad<VB> q[U];
    auto load = [&](int i0, int u0) {
#pragma unroll
      for (int u = u0; u < u0 + U / 2; ++u) {
        q[u].zero();
        if (i0 + u < nv) q[u].load(v + (long long)(i0 + u) * N, n4);
      }
    };
    load(0, 0);
    for (int i0 = 0; i0 < nv; i0 += U) {
      load(i0, U / 2);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float2 h = hs[i0 + u];
#pragma unroll
        for (int r = 0; r < 4; ++r) cms(acc[r], q[u].get(r), h);
        if (u == U / 2 - 1) load(i0 + U, 0);
      }
    }
    wp[0] = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    wp[1] = make_float4(acc[2].x, acc[2].y, acc[3].x, acc[3].y);
    if (MODE) {
      AccF32 f;
#pragma unroll
      for (int r = 0; r < 4; ++r) f.add_norm(acc[r]);
      nrm2 += (double)f.re;
    }
  }
  AccF32 a;
  a.re = (float)nrm2;
  if constexpr (MODE >= 1) update_tail<MODE>(a, b, nrm_partial, nv, pstride, nblk, tl);
}

// The same in FP64: one complex value per thread, bound by the FP64 pipe (4 FMAs per element and vector).
// Explicit FMAs: w -= v h had compiled to a multiply, an FMA and a subtraction per component.  2 problems of
// 245,760 unknowns, 25 vectors: 156 -> 96 us (0.94 TFLOP/s).
template <int MODE>
__global__ void __launch_bounds__(256) gs_update64_kernel(const double2* __restrict__ V, double2* __restrict__ w,
                                                          const double2* __restrict__ hcol,
                                                          const int* __restrict__ mask,
                                                          double* __restrict__ nrm_partial, long long N, int nv,
                                                          int mp1, int pstride, int nblk, KrylovTail tl) {
  const int b = blockIdx.y;
  if (!mask[b]) return;
  __shared__ double2 hs[kMaxRestart + 1];
  for (int i = threadIdx.x; i < nv; i += blockDim.x) hs[i] = hcol[b * pstride + i];
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long t = (long long)b * N + n;
  double2 acc = n < N ? w[t] : make_double2(0.0, 0.0);
  __syncthreads();
  Acc64 a;
  if (n < N) {
    const double2* v = V + (long long)b * mp1 * N + n;
#pragma unroll 8
    for (int i = 0; i < nv; ++i) cms(acc, __ldg(v + (long long)i * N), hs[i]);
    w[t] = acc;
    if (MODE) a.add_norm(acc);
  }
  if constexpr (MODE >= 1) update_tail<MODE>(a, b, nrm_partial, nv, pstride, nblk, tl);
}

template <typename T>
__global__ void __launch_bounds__(256) norm_partial_kernel(const T* __restrict__ v, double* __restrict__ out,
                                                           long long N, int nchunk,
                                                           const int* __restrict__ mask = nullptr) {
  const int b = blockIdx.y, c = blockIdx.x;
  if (mask && !mask[b]) return;
  const T* vv = v + (long long)b * N;
  typename AccFor<T>::type a;
  for (long long n = (long long)c * 256 + threadIdx.x; n < N; n += (long long)nchunk * 256) a.add_norm(vv[n]);
  const double acc = block_sum1(a.get().x);
  if (threadIdx.x == 0) out[b * nchunk + c] = acc;
}

// out[b] = sqrt(sum_c partial); optionally H[b][k][k+1] = out[b]
__global__ void norm_reduce_kernel(const double* __restrict__ partial, double* __restrict__ out,
                                   double2* __restrict__ H, const int* __restrict__ active, int nchunk, int k,
                                   int pstride, int m, double* __restrict__ inv64 = nullptr,
                                   float* __restrict__ inv32 = nullptr, const int* __restrict__ mask = nullptr) {
  const int b = blockIdx.x;
  if (mask && !mask[b]) return;   // problems outside the mask keep their norm
  double acc = 0;
  for (int c = threadIdx.x; c < nchunk; c += 32) acc += partial[b * nchunk + c];
  acc = warp_sum(acc);
  if (threadIdx.x == 0) {
    const double v = sqrt(acc);
    out[b] = v;
    if (inv64) inv64[b] = v > 0 ? 1.0 / v : 0.0;
    if (inv32) inv32[b] = v > 0 ? (float)(1.0 / v) : 0.f;
    if (H && active[b]) H[(long long)b * pstride * m + (long long)k * pstride + k + 1] = make_double2(v, 0.0);
  }
}

// dst = src * inv[b]  (inverse norms precomputed per problem)
template <typename S, typename D>
__global__ void __launch_bounds__(256) scale_kernel(const S* __restrict__ src, D* __restrict__ dst,
                                                    const double* __restrict__ nrm, const int* __restrict__ active,
                                                    long long N, long long dst_stride, int batch) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * batch) return;
  const int b = (int)(t / N);
  if (!active[b]) return;
  const long long n = t - (long long)b * N;
  const double inv = nrm[b];   // inverse norm
  const double2 v = ld2(src[t]);
  st2(dst[(long long)b * dst_stride + n], make_double2(v.x * inv, v.y * inv));
}

__global__ void __launch_bounds__(256) residual_kernel(const double2* __restrict__ rhs, const double2* __restrict__ ax,
                                                       double2* __restrict__ r, long long total, long long N,
                                                       const int* __restrict__ mask) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total || (mask && !mask[t / N])) return;
  const double2 a = rhs[t], b = ax[t];
  r[t] = make_double2(a.x - b.x, a.y - b.y);
}

// x += s[b] * z  (s = nullptr: s = 1; problems with mask[b] == 0 are left as they are)
template <typename T>
__global__ void __launch_bounds__(256) axpy_kernel(double2* __restrict__ x, const T* __restrict__ z,
                                                   const double* __restrict__ s, long long N, int batch,
                                                   const int* __restrict__ mask = nullptr) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * batch) return;
  const int b = (int)(t / N);
  if (mask && !mask[b]) return;
  const double f = s ? s[b] : 1.0;
  const double2 a = x[t], v = ld2(z[t]);
  x[t] = make_double2(a.x + f * v.x, a.y + f * v.y);
}

__global__ void cycle_init_kernel(const double* __restrict__ nrm, const double* __restrict__ target,
                                  double2* __restrict__ g, int* __restrict__ active, int* __restrict__ kused,
                                  int pstride, int batch) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  const double beta = nrm[b];
  const int act = (beta > target[b]) && isfinite(beta);
  active[b] = act;
  kused[b] = 0;
  for (int i = 0; i < pstride; ++i) g[b * pstride + i] = make_double2(i == 0 ? beta : 0.0, 0.0);
}


template <typename T, typename VB = T>
__global__ void __launch_bounds__(256) combine_kernel(const VB* __restrict__ V, const T* __restrict__ y,
                                                      const int* __restrict__ kused, T* __restrict__ u, long long N,
                                                      int mp1, int m, int batch) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * batch) return;
  const int b = (int)(t / N);
  const long long n = t - (long long)b * N;
  const int kk = kused[b];
  T acc;
  acc.x = 0;
  acc.y = 0;
  const VB* v = V + (long long)b * mp1 * N + n;
  for (int i = 0; i < kk; ++i) {
    T h = y[b * m + i];
    h.x = -h.x;
    h.y = -h.y;
    cms(acc, ld_one(v[(long long)i * N]), h);   // acc += v y
  }
  u[t] = acc;
}

inline unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

#define WG_CK(expr)                                                        \
  do {                                                                     \
    cudaError_t e_ = (expr);                                               \
    if (e_ != cudaSuccess) {                                               \
      P.err = std::string("CUDA: ") + cudaGetErrorString(e_) + " at " #expr; \
      return WG_ERR_CUDA;                                                  \
    }                                                                      \
  } while (0)

// One Arnoldi step k on basis V (stride (m+1) N per problem): z = M^-1 V_k,
// w = A z, CGS2 against V_0..V_k, V_{k+1} = w / |w|, Givens.  `prec` and `apply`
// are the operator pair of the basis precision.
template <typename T> float2* coef_col32(Problem& P);
template <> float2* coef_col32<double2>(Problem&) { return nullptr; }
template <> float2* coef_col32<float2>(Problem& P) { return P.mx.hcol; }

template <typename T, typename VB = T, typename Prec, typename Apply>
int arnoldi_step(Problem& P, VB* V, T* w, int k, int m, bool pre, Prec prec, Apply apply) {
  const int B = P.batch, mp1 = m + 1, ps = P.restart_max + 1, mm = P.restart_max;
  const long long N = P.N;
  // V_k: step 0 reads the basis vector the cycle start wrote; later steps take the previous
  // step's w and its inverse norm, and the preconditioner writes V_k = w / |w| as it reads it
  // (no separate scaling pass per step).  An FP16 basis: the cycle start leaves V_0 in FP32
  // in w, and the preconditioner stores its FP16 rounding as V_0.
  if (k == 0) {
    if constexpr (std::is_same<VB, T>::value) WG_CK(prec(V, (long long)mp1 * N, nullptr, nullptr));
    else WG_CK(prec(w, N, nullptr, V));
  } else {
    const T* wprev = w;
    if constexpr (std::is_same<T, float2>::value)
      WG_CK(prec(wprev, N, P.mx.inv, V + (long long)k * N));
    else
      WG_CK(prec(wprev, N, P.inv64, V + (long long)k * N));
  }
  WG_CK(apply(V + (long long)k * N));
  const int nv = k + 1;
  const double vec = (double)N * B * sizeof(T), vecb = (double)N * B * sizeof(VB);
  constexpr bool f32 = std::is_same<T, float2>::value;
  const int mq = dot_quads(N), uq = update_quads(N);
  const int mblk = (int)((N / 4 + mq - 1) / mq);
  const int nblk = f32 ? (int)((N / 4 + uq - 1) / uq) : (int)((N + 255) / 256);
  const dim3 gu(nblk, B);
  // classical Gram-Schmidt; the second pass runs for the problems that fail the DGKS
  // test (its kernels see P.reorth as their activity mask), for all with eta >= 1,
  // for none with eta < 0.  The reductions, the norm and the Givens step run in the
  // last block of each problem's multi-dot / update launch (KrylovTail).
  const double eta = sizeof(T) == sizeof(float2) ? P.inner_reorth_eta : P.reorth_eta;
  const int passes = eta < 0 ? 1 : 2;
  KrylovTail tl{P.md_count, P.gs_count, P.partial, P.hcol, coef_col32<T>(P), P.H, P.cs, P.sn, P.g, P.active,
                P.kused, P.reorth, P.target, P.nrm, sizeof(T) == sizeof(float2) ? nullptr : P.inv64,
                sizeof(T) == sizeof(float2) ? P.mx.inv : nullptr, eta * eta, pre ? 1.0 : 0.0, k, ps, mm, 1};
  // the DGKS flags are written only for problems that take part in the first pass
  if (passes == 2 && eta < 1) WG_CK(cudaMemsetAsync(P.reorth, 0, sizeof(int) * B, P.stream));
  for (int pass = 0; pass < passes; ++pass) {
    const int* mask = (pass == 0 || eta >= 1) ? P.active : P.reorth;
    tl.first = pass == 0;
    cudaEvent_t ev = prof_begin(P, PROF_MULTIDOT, 1, nv * vecb + vec, 8.0 * nv * N * B, mask);
    if constexpr (f32) {
      multidot32_kernel<VB><<<dim3(mblk, B), 256, sizeof(double) * 16 * ((nv + 3) & ~3), P.stream>>>(
          V, w, P.partial, mask, N, nv, mp1, ps, mblk, mq, tl);
    } else {
      const dim3 gm(P.md_chunk, B, (nv + 3) / 4);
      auto md = P.md_e == 8 ? multidot64_kernel<8> : P.md_e == 4 ? multidot64_kernel<4>
                                                   : P.md_e == 2 ? multidot64_kernel<2> : multidot64_kernel<1>;
      md<<<gm, 256, 0, P.stream>>>(V, w, P.partial, mask, N, nv, mp1, ps, P.md_chunk, tl);
    }
    prof_end(P, PROF_MULTIDOT, ev);
    ev = prof_begin(P, PROF_GSUPDATE, 1, nv * vecb + 2 * vec, 8.0 * nv * N * B, mask);
    const int mode = pass == passes - 1 ? 2 : (eta < 1 ? 1 : 0);
    if constexpr (f32) {
      auto up = mode == 2 ? gs_update32_kernel<2, VB> : mode == 1 ? gs_update32_kernel<1, VB>
                                                                  : gs_update32_kernel<0, VB>;
      up<<<gu, kUp32Threads, 0, P.stream>>>(V, w, P.mx.hcol, mask, P.nrm_partial, N, nv, mp1, ps, nblk, uq, tl);
    } else {
      auto up = mode == 2 ? gs_update64_kernel<2> : mode == 1 ? gs_update64_kernel<1> : gs_update64_kernel<0>;
      up<<<gu, 256, 0, P.stream>>>(V, w, P.hcol, mask, P.nrm_partial, N, nv, mp1, ps, nblk, tl);
    }
    prof_end(P, PROF_GSUPDATE, ev);
  }
  // V_{k+1} = w / |w| is written by the next step's preconditioner
  WG_CK(cudaGetLastError());
  return WG_OK;
}

constexpr int kResidualDigits = 7;   // of the emulated FP64 transforms in the mixed form's residual (digits_for)

// r = rhs - A x ; nrm[b] = |r_b|  (FP64)
// r = b - A x and |r| (FP64; the mixed form's transforms on the tensor cores).  mask
// (device, optional): only problems with mask[b] != 0 are evaluated, the others keep
// their previous r and |r| (their x has not changed since).
int true_residual(Problem& P, const int* mask = nullptr, int nd = kResidualDigits, const int* nd_pp = nullptr) {
  const long long tot = P.N * P.batch;
  P.prof.launches[PROF_OTHER] += 3;
  if (P.precision == WG_PREC_MIXED) WG_CK(launch_apply_f64_tc(P, P.x, P.w, mask, nd, nd_pp));
  else WG_CK(launch_apply(P, P.x, P.w));
  residual_kernel<<<blocks_for(tot), 256, 0, P.stream>>>(P.rhs, P.w, P.r, tot, P.N, mask);
  norm_partial_kernel<double2><<<dim3(P.nchunk, P.batch), 256, 0, P.stream>>>(P.r, P.nrm_partial, P.N, P.nchunk,
                                                                             mask);
  norm_reduce_kernel<<<P.batch, 32, 0, P.stream>>>(P.nrm_partial, P.nrm, nullptr, P.active, P.nchunk, 0, 0, 0,
                                                   P.inv64, nullptr, mask);
  WG_CK(cudaGetLastError());
  return WG_OK;
}

// Leading digits of the emulated FP64 transforms for the mixed form's true residual: enough
// that the residual's error (~2^(-7 nd) |A||x|, with a margin of 2^21 for |A||x| / |b|) stays
// below the loosest target among the problems it is evaluated for; 7 (49 bits) for
// tolerances of 1e-6 and below.  WG_RESIDUAL_DIGITS (1 .. 8) fixes it.
int digits_for(double t) {
  if (!(t > 0) || !(t < 1e299)) return kResidualDigits;
  const int d = (int)std::ceil((std::log2(1.0 / t) + 21.0) / 7.0);
  return std::max(4, std::min(kResidualDigits, d));
}

int residual_digits(const Problem& P, double tol, const std::vector<int>* hmask) {
  static const int forced = [] {
    const char* v = std::getenv("WG_RESIDUAL_DIGITS");
    const int d = v ? std::atoi(v) : 0;
    return (d >= 1 && d <= 8) ? d : 0;
  }();
  if (forced) return forced;
  double tmin = INFINITY;
  for (int b = 0; b < P.batch; ++b) {
    if (hmask && (int)hmask->size() == P.batch && !(*hmask)[b]) continue;
    tmin = std::min(tmin, P.tol_pp.empty() ? tol : P.tol_pp[b]);
  }
  return digits_for(tmin);
}

// Digits per problem (the emulated GEMM's column tiles take the largest of their problems);
// uploads them and returns the device array, or nullptr when one count serves all.
const int* residual_digits_pp(Problem& P, double tol) {
  if (P.tol_pp.empty() || std::getenv("WG_RESIDUAL_DIGITS")) return nullptr;
  P.h_res_digits.assign(P.batch, kResidualDigits);
  for (int b = 0; b < P.batch; ++b) P.h_res_digits[b] = digits_for(P.tol_pp[b]);
  if (cudaMemcpyAsync(P.res_digits, P.h_res_digits.data(), sizeof(int) * P.batch, cudaMemcpyHostToDevice,
                      P.stream) != cudaSuccess)
    return nullptr;
  return P.res_digits;
}

// Shared set-up: |b| per problem, targets, initial true residual.
int solve_begin(Problem& P, double tol, bool warm, std::vector<double>& bnorm, std::vector<double>& tgt,
                std::vector<double>& res) {
  const int B = P.batch;
  if (!warm) WG_CK(cudaMemsetAsync(P.x, 0, sizeof(double2) * P.N * B, P.stream));
  P.prof.launches[PROF_OTHER] += 2;
  norm_partial_kernel<double2><<<dim3(P.nchunk, B), 256, 0, P.stream>>>(P.rhs, P.nrm_partial, P.N, P.nchunk);
  norm_reduce_kernel<<<B, 32, 0, P.stream>>>(P.nrm_partial, P.nrm, nullptr, P.active, P.nchunk, 0, 0, 0);
  bnorm.resize(B);
  WG_CK(cudaMemcpyAsync(bnorm.data(), P.nrm, sizeof(double) * B, cudaMemcpyDeviceToHost, P.stream));
  WG_CK(cudaStreamSynchronize(P.stream));
  tgt.resize(B);
  for (int b = 0; b < B; ++b) tgt[b] = (P.tol_pp.empty() ? tol : P.tol_pp[b]) * bnorm[b];
  // problems frozen by an unreachable tolerance keep their residual
  const int* mask = nullptr;
  int nd = kResidualDigits;
  if (P.precision == WG_PREC_MIXED) {
    if (!P.tol_pp.empty()) {
      P.h_res_mask.assign(B, 1);
      for (int b = 0; b < B; ++b) P.h_res_mask[b] = P.tol_pp[b] < 1e299 ? 1 : 0;
      WG_CK(cudaMemcpyAsync(P.res_mask, P.h_res_mask.data(), sizeof(int) * B, cudaMemcpyHostToDevice, P.stream));
      mask = P.res_mask;
      nd = residual_digits(P, tol, &P.h_res_mask);
    } else {
      nd = residual_digits(P, tol, nullptr);
    }
  }
  int rc = true_residual(P, mask, nd, P.precision == WG_PREC_MIXED ? residual_digits_pp(P, tol) : nullptr);
  if (rc) return rc;
  res.resize(B);
  WG_CK(cudaMemcpyAsync(res.data(), P.nrm, sizeof(double) * B, cudaMemcpyDeviceToHost, P.stream));
  WG_CK(cudaStreamSynchronize(P.stream));
  return WG_OK;
}

int solve_end(Problem& P, const std::vector<double>& bnorm, const std::vector<double>& tgt,
              const std::vector<double>& initial, const std::vector<double>& res, const std::vector<int>& iters,
              const std::vector<int>& cycles, const std::vector<int>& refinements, wg_solve_info* info) {
  int status = WG_OK;
  for (int b = 0; b < P.batch; ++b) {
    wg_solve_info& in = info[b];
    const double bn = bnorm[b] > 0 ? bnorm[b] : 1.0;
    in.rhs_norm = bnorm[b];
    in.relres = res[b] / bn;
    in.initial_relres = initial[b] / bn;
    in.iterations = iters[b];
    in.cycles = cycles[b];
    in.refinements = refinements[b];
    in.flag = (std::isfinite(res[b]) && res[b] <= tgt[b]) ? 0 : 1;
    if (bnorm[b] == 0) in.flag = 0;
    if (!std::isfinite(res[b])) {
      P.err = "non-finite residual (NaN/Inf in operator data or rhs)";
      status = WG_ERR_NUMERIC;
    }
    if (in.flag && status == WG_OK) status = WG_NOT_CONVERGED;
  }
  return status;
}

bool all_done(const std::vector<int>& act) {
  for (int a : act)
    if (a) return false;
  return true;
}

bool graphs_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("WG_CUDA_GRAPHS");
    return !(v && v[0] == '0');
  }();
  return on;
}

void reset_graphs(ArnoldiGraphs& G) {
  for (cudaGraphExec_t x : G.exec)
    if (x) cudaGraphExecDestroy(x);
  G.exec.clear();
  G.launches.clear();
  G.eager.clear();
}

// Arnoldi steps k0 .. k0+3 (fewer at the end of the cycle) of a cycle of length m, run
// eagerly (`run`) or replayed from the chunk's CUDA graph.  A chunk is captured on its
// second use, so the launch helpers' one-time set-up has run outside the capture; any
// failure to capture or instantiate falls back to eager launches for the handle.
// Chunks of a cycle: steps [0,1), [1,2), [2,4), then 4 at a time.  The host checks the
// problems' convergence after every chunk; the short first chunks keep a cycle that
// converges in one or two steps (loose transport tolerances) from running masked steps.
int chunk_end(int k0, int m) { return std::min(m, k0 < 2 ? k0 + 1 : (k0 < 4 ? 4 : k0 + 4)); }
int chunk_index(int k0) { return k0 < 2 ? k0 : (k0 < 4 ? 2 : 2 + k0 / 4); }
int chunk_count(int m) { return m <= 2 ? m : (m <= 4 ? 3 : 2 + (m + 3) / 4); }

template <typename Run>
int run_arnoldi_chunk(Problem& P, ArnoldiGraphs& G, int m, int k0, Run run) {
  if (G.disabled || P.prof.on || !graphs_enabled()) return run();
  const int nchunk = chunk_count(m), c = chunk_index(k0);
  if (G.m != m || G.shift != P.shift || G.kline_L != P.kline_L || G.st_cells != P.st_cells ||
      (int)G.exec.size() != nchunk) {
    reset_graphs(G);
    G.m = m;
    G.shift = P.shift;
    G.kline_L = P.kline_L;
    G.st_cells = P.st_cells;
    G.exec.assign(nchunk, nullptr);
    G.launches.assign(nchunk, {});
    G.eager.assign(nchunk, 0);
  }
  if (G.exec[c]) {
    const cudaError_t e = cudaGraphLaunch(G.exec[c], P.stream);
    if (e != cudaSuccess) {
      P.err = std::string("CUDA graph launch: ") + cudaGetErrorString(e);
      return WG_ERR_CUDA;
    }
    for (int i = 0; i < PROF_N; ++i) P.prof.launches[i] += G.launches[c][i];
    ++G.replays;
    return WG_OK;
  }
  if (G.eager[c]++ == 0) return run();
  std::array<long long, PROF_N> before;
  for (int i = 0; i < PROF_N; ++i) before[i] = P.prof.launches[i];
  auto fall_back = [&]() {
    cudaGetLastError();
    G.disabled = true;
    reset_graphs(G);
    for (int i = 0; i < PROF_N; ++i) P.prof.launches[i] = before[i];
    return run();
  };
  if (cudaStreamBeginCapture(P.stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return fall_back();
  const int rc = run();
  cudaGraph_t g = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(P.stream, &g);
  if (rc != WG_OK || ec != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    return fall_back();
  }
  cudaGraphExec_t x = nullptr;
  const cudaError_t ei = cudaGraphInstantiate(&x, g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess || !x) return fall_back();
  G.exec[c] = x;
  for (int i = 0; i < PROF_N; ++i) G.launches[c][i] = P.prof.launches[i] - before[i];
  const cudaError_t e = cudaGraphLaunch(x, P.stream);
  if (e != cudaSuccess) {
    P.err = std::string("CUDA graph launch: ") + cudaGetErrorString(e);
    return WG_ERR_CUDA;
  }
  return WG_OK;
}

}  // namespace

int gmres_solve_fp64(Problem& P, const wg_solve_opts& o, bool warm, wg_solve_info* info) {
  const int B = P.batch, m = P.restart, mp1 = m + 1, ps = P.restart_max + 1, mm = P.restart_max;
  const long long N = P.N, tot = N * B;
  const double tol = o.tol > 0 ? o.tol : 1e-10;
  const int maxit = o.maxit > 0 ? o.maxit : 50;
  std::vector<double> bnorm, tgt, initial;
  int rc = solve_begin(P, tol, warm, bnorm, tgt, initial);
  if (rc) return rc;
  WG_CK(cudaMemcpyAsync(P.target, tgt.data(), sizeof(double) * B, cudaMemcpyHostToDevice, P.stream));
  std::vector<int> iters(B, 0), cycles(B, 0), refs(B, 0);
  std::vector<double> res = initial;
  auto prec = [&](const double2* r, long long stride, const double* rscale, double2* rout) {
    return launch_precondition(P, r, stride, P.z, rscale, rout, (long long)mp1 * N);
  };
  const bool pre = flux_is_inverted(P);
  auto apply = [&](const double2* v) {
    return pre ? launch_apply_pre(P, P.z, v, (long long)mp1 * N, P.w) : launch_apply(P, P.z, P.w);
  };
  for (int cyc = 0; cyc < maxit; ++cyc) {
    bool any = false;
    for (int b = 0; b < B; ++b) any |= (res[b] > tgt[b]) && std::isfinite(res[b]);
    if (!any) break;
    P.prof.launches[PROF_OTHER] += 2;
    cycle_init_kernel<<<(B + 127) / 128, 128, 0, P.stream>>>(P.nrm, P.target, P.g, P.active, P.kused, ps, B);
    scale_kernel<double2, double2><<<blocks_for(tot), 256, 0, P.stream>>>(P.r, P.V, P.inv64, P.active, N,
                                                                         (long long)mp1 * N, B);
    for (int k0 = 0; k0 < m; k0 = chunk_end(k0, m)) {
      const int k1 = chunk_end(k0, m);
      rc = run_arnoldi_chunk(P, P.graphs[0], m, k0, [&]() {
        for (int k = k0; k < k1; ++k) {
          const int r = arnoldi_step<double2>(P, P.V, P.w, k, m, pre, prec, apply);
          if (r) return r;
        }
        return (int)WG_OK;
      });
      if (rc) return rc;
      WG_CK(cudaMemcpyAsync(P.h_active.data(), P.active, sizeof(int) * B, cudaMemcpyDeviceToHost, P.stream));
      WG_CK(cudaStreamSynchronize(P.stream));
      if (all_done(P.h_active)) break;
    }
    P.prof.launches[PROF_OTHER] += 3;
    backsolve_kernel<<<B, 32, 0, P.stream>>>(P.H, P.g, P.ycoef, nullptr, P.kused, ps, mm, B);
    combine_kernel<double2><<<blocks_for(tot), 256, 0, P.stream>>>(P.V, P.ycoef, P.kused, P.w, N, mp1, mm, B);
    WG_CK(launch_precondition(P, P.w, N, P.z));
    axpy_kernel<double2><<<blocks_for(tot), 256, 0, P.stream>>>(P.x, P.z, nullptr, N, B);
    WG_CK(cudaGetLastError());
    rc = true_residual(P);
    if (rc) return rc;
    WG_CK(cudaMemcpyAsync(P.h_kused.data(), P.kused, sizeof(int) * B, cudaMemcpyDeviceToHost, P.stream));
    WG_CK(cudaMemcpyAsync(res.data(), P.nrm, sizeof(double) * B, cudaMemcpyDeviceToHost, P.stream));
    WG_CK(cudaStreamSynchronize(P.stream));
    for (int b = 0; b < B; ++b) {
      iters[b] += P.h_kused[b];
      if (P.h_kused[b] > 0) cycles[b] += 1;
    }
  }
  rc = tc_status(P, "wg_solve");
  if (rc) return rc;
  return solve_end(P, bnorm, tgt, initial, res, iters, cycles, refs, info);
}

// FP64 iterative refinement around one FP32/BF16 GMRES cycle per correction.
int gmres_solve_mixed(Problem& P, const wg_solve_opts& o, bool warm, wg_solve_info* info) {
  const int B = P.batch, m = P.restart_inner, mp1 = m + 1, ps = P.restart_max + 1, mm = P.restart_max;
  const long long N = P.N, tot = N * B;
  const double tol = o.tol > 0 ? o.tol : 1e-10;
  const int max_ref = o.maxit > 0 ? o.maxit : 50;
  MixedBuffers& M = P.mx;
  WG_CK(mixed_sync_weights(P));
  std::vector<double> bnorm, tgt, initial;
  int rc = solve_begin(P, tol, warm, bnorm, tgt, initial);
  if (rc) return rc;
  std::vector<int> iters(B, 0), cycles(B, 0), refs(B, 0);
  std::vector<double> res = initial, itgt(B), ones(B, 1.0);
  // with the flux inverted by the preconditioner only z's BF16 copy is needed
  const bool pre = flux_is_inverted(P) && !M.fused;
  float2* zf = pre ? nullptr : M.z;
  // the inner Arnoldi steps skip problems that have converged in this cycle (P.active)
  auto prec = [&](const float2* r, long long stride, const float* rscale, float2* rout) {
    return launch_precondition_mixed(P, r, stride, zf, M.zb16, P.active, rscale, rout, (long long)mp1 * N);
  };
  auto prec_h = [&](const float2* r, long long stride, const float* rscale, __half2* rout) {
    return launch_precondition_mixed_h(P, r, stride, zf, M.zb16, P.active, rscale, rout, (long long)mp1 * N);
  };
  auto apply = [&](const auto*) {
    return pre ? launch_apply_mixed_pre(P, M.w, P.active) : launch_apply_mixed(P, M.z, M.zb16, M.w, P.active);
  };
  for (int ref = 0; ref < max_ref; ++ref) {
    bool any = false;
    for (int b = 0; b < B; ++b) any |= (res[b] > tgt[b]) && std::isfinite(res[b]);
    if (!any) break;
    // inner target on the normalised residual: reach the outer target, never below inner_tol
    P.h_res_mask.assign(B, 0);
    for (int b = 0; b < B; ++b) {
      const bool act = (res[b] > tgt[b]) && std::isfinite(res[b]);
      itgt[b] = act ? std::max(P.inner_tol, 0.5 * tgt[b] / res[b]) : INFINITY;
      P.h_res_mask[b] = act ? 1 : 0;
    }
    WG_CK(cudaMemcpyAsync(P.target, itgt.data(), sizeof(double) * B, cudaMemcpyHostToDevice, P.stream));
    WG_CK(cudaMemcpyAsync(P.res_mask, P.h_res_mask.data(), sizeof(int) * B, cudaMemcpyHostToDevice, P.stream));
    // keep |r| for the update, start the inner cycle from the unit-norm residual
    WG_CK(cudaMemcpyAsync(P.nrm_keep, P.nrm, sizeof(double) * B, cudaMemcpyDeviceToDevice, P.stream));
    WG_CK(cudaMemcpyAsync(P.nrm, ones.data(), sizeof(double) * B, cudaMemcpyHostToDevice, P.stream));
    P.prof.launches[PROF_OTHER] += 2;
    cycle_init_kernel<<<(B + 127) / 128, 128, 0, P.stream>>>(P.nrm, P.target, P.g, P.active, P.kused, ps, B);
    // V_0 = r / |r| (an FP16 basis: in FP32 in w, stored by the first step's preconditioner)
    if (M.basis16)
      scale_kernel<double2, float2><<<blocks_for(tot), 256, 0, P.stream>>>(P.r, M.w, P.inv64, P.active, N, N, B);
    else
      scale_kernel<double2, float2><<<blocks_for(tot), 256, 0, P.stream>>>(P.r, M.V, P.inv64, P.active, N,
                                                                          (long long)mp1 * N, B);
    for (int k0 = 0; k0 < m; k0 = chunk_end(k0, m)) {
      const int k1 = chunk_end(k0, m);
      rc = run_arnoldi_chunk(P, P.graphs[1], m, k0, [&]() {
        for (int k = k0; k < k1; ++k) {
          const int r = M.basis16 ? arnoldi_step<float2, __half2>(P, M.Vh, M.w, k, m, pre, prec_h, apply)
                                  : arnoldi_step<float2>(P, M.V, M.w, k, m, pre, prec, apply);
          if (r) return r;
        }
        return (int)WG_OK;
      });
      if (rc) return rc;
      WG_CK(cudaMemcpyAsync(P.h_active.data(), P.active, sizeof(int) * B, cudaMemcpyDeviceToHost, P.stream));
      WG_CK(cudaStreamSynchronize(P.stream));
      if (all_done(P.h_active)) break;
    }
    // d = M^-1 (V y) in FP32, x += |r| d in FP64
    P.prof.launches[PROF_OTHER] += 3;
    backsolve_kernel<<<B, 32, 0, P.stream>>>(P.H, P.g, P.ycoef, M.y, P.kused, ps, mm, B);
    if (M.basis16)
      combine_kernel<float2, __half2><<<blocks_for(tot), 256, 0, P.stream>>>(M.Vh, M.y, P.kused, M.w, N, mp1, mm, B);
    else
      combine_kernel<float2><<<blocks_for(tot), 256, 0, P.stream>>>(M.V, M.y, P.kused, M.w, N, mp1, mm, B);
    WG_CK(launch_precondition_mixed(P, M.w, N, M.d, nullptr, P.res_mask));
    axpy_kernel<float2><<<blocks_for(tot), 256, 0, P.stream>>>(P.x, M.d, P.nrm_keep, N, B, P.res_mask);
    WG_CK(cudaGetLastError());
    // problems that did not move this refinement keep r and |r|; the others are re-evaluated
    WG_CK(cudaMemcpyAsync(P.nrm, P.nrm_keep, sizeof(double) * B, cudaMemcpyDeviceToDevice, P.stream));
    rc = true_residual(P, P.res_mask, residual_digits(P, tol, &P.h_res_mask), residual_digits_pp(P, tol));
    if (rc) return rc;
    int herr = 0;
    WG_CK(cudaMemcpyAsync(&herr, M.err, sizeof(int), cudaMemcpyDeviceToHost, P.stream));
    WG_CK(cudaMemcpyAsync(P.h_kused.data(), P.kused, sizeof(int) * B, cudaMemcpyDeviceToHost, P.stream));
    WG_CK(cudaMemcpyAsync(res.data(), P.nrm, sizeof(double) * B, cudaMemcpyDeviceToHost, P.stream));
    WG_CK(cudaStreamSynchronize(P.stream));
    if (herr) {
      P.err = "tensor-core GEMM: bounded barrier wait timed out";
      return WG_ERR_TIMEOUT;
    }
    for (int b = 0; b < B; ++b) {
      iters[b] += P.h_kused[b];
      if (P.h_kused[b] > 0) {
        cycles[b] += 1;
        refs[b] += 1;
      }
    }
  }
  WG_CK(cudaMemcpyAsync(P.target, tgt.data(), sizeof(double) * B, cudaMemcpyHostToDevice, P.stream));
  WG_CK(cudaStreamSynchronize(P.stream));
  return solve_end(P, bnorm, tgt, initial, res, iters, cycles, refs, info);
}

int solve_dispatch(Problem& P, const wg_solve_opts& o, bool warm, wg_solve_info* info) {
  if (!P.tuned) {
    const int rt = autotune(P);
    if (rt) return rt;
  }
  if (P.precision == WG_PREC_MIXED) return gmres_solve_mixed(P, o, warm, info);
  return gmres_solve_fp64(P, o, warm, info);
}

}  // namespace wg
