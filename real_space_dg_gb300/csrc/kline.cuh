// k-line preconditioner sweep over (k line, element chunk, problem).
//
// In 1D the flux operator of wave number k is block-bidiagonal over the elements
// with an upwind coupling that touches one node of the neighbour element
// (get_LineTransversePreconditioner_full2D.m:174-239 reduced to one line per k):
//   z_e = D_b(k) r_e / qd_b - h_b(k) s_{e-1},   s_e = z_e[st]
// (st = the last local node for k > 0, sweeping e upwards; the first for k < 0,
// sweeping downwards).  The scalar recurrence s_e = a s_{e-1} + c_e is affine, so
// the elements are cut into chunks of L:
//   kline_maps_kernel   each (k, chunk) composes its chunk's map s -> A s + S from a
//                       zero start (one pass over the chunk's r);
//   kline_apply_kernel  each (k, chunk) folds the maps of the chunks upwind of it
//                       into its incoming s, then sweeps its chunk writing z.
// Threads: x = 32 consecutive k (coalesced rows), y = 4 chunks; grid
// (ceil(nk/32), ceil(n_chunks/4), batch) covers every SM even for one problem.
// Chunks of up to FusedLen elements take one launch instead (kline_fused_kernel): all chunks of a few lines in
// one block, each thread's chunk of r in registers from its only read on, the maps in shared memory.
// Optional: r enters scaled by rscale[b] (the Arnoldi step's w / |w|), and the apply kernel
// writes the scaled r to rout (the next basis vector), which replaces a separate scaling pass.
// With an FP16 basis (rout of type __half2) both kernels round the scaled r to FP16 before
// they use it, so z is the preconditioned image of exactly the stored basis vector.  z may be null where the
// BF16 copy zb alone is used.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include <vector>

namespace wg {
namespace kline {

constexpr int kChunksPerBlock = 4;

template <typename R> struct Cplx;
template <> struct Cplx<double> { using type = double2; };
template <> struct Cplx<float> { using type = float2; };

__device__ __forceinline__ double rcp(double x) { return 1.0 / x; }
__device__ __forceinline__ float rcp(float x) { return __frcp_rn(x); }

// r value as the basis stores it: unchanged, or rounded to FP16 (RH)
template <bool RH, typename T>
__device__ __forceinline__ T basis_round(T v) {
  if constexpr (RH) {
    const float2 f = __half22float2(__floats2half2_rn((float)v.x, (float)v.y));
    v.x = f.x;
    v.y = f.y;
  }
  return v;
}
__device__ __forceinline__ void basis_store(float2& d, float2 v) { d = v; }
__device__ __forceinline__ void basis_store(double2& d, double2 v) { d = v; }
__device__ __forceinline__ void basis_store(__half2& d, float2 v) { d = __floats2half2_rn(v.x, v.y); }

template <int NK, typename R, bool RH = false>
__global__ void __launch_bounds__(32 * kChunksPerBlock) kline_maps_kernel(
    const typename Cplx<R>::type* __restrict__ r, const R* __restrict__ kvec, const R* __restrict__ dinv,
    const R* __restrict__ hvec, const R* __restrict__ qd, R* __restrict__ mapA, typename Cplx<R>::type* __restrict__ mapS,
    int n_el, int nk, long long N, long long r_stride, int L, int nchunk, const int* __restrict__ mask,
    const R* __restrict__ rscale = nullptr) {
  using T = typename Cplx<R>::type;
  const int j = blockIdx.x * 32 + threadIdx.x;
  const int c = blockIdx.y * kChunksPerBlock + threadIdx.y;
  const int b = blockIdx.z;
  if (j >= nk || c >= nchunk || (mask && !mask[b])) return;
  const long long bj = (long long)b * nk + j;
  const bool fwd = kvec[j] > R(0);
  const int st = fwd ? NK - 1 : 0;
  const R sc = rscale ? rscale[b] : R(1);   // r enters scaled (the basis vector w / |w|)
  R Dst[NK];
#pragma unroll
  for (int q = 0; q < NK; ++q) Dst[q] = dinv[bj * NK * NK + st * NK + q];
  const R alpha = -hvec[bj * NK + st];
  const R inv_qd = qd[b] > R(0) ? rcp(qd[b]) : R(0);   // a problem without data stays zero
  const int e_lo = c * L, e_hi = min(n_el, e_lo + L);
  const T* rb = r + (long long)b * r_stride + j;
  R A = R(1);
  T s;
  s.x = R(0);
  s.y = R(0);
  for (int i = 0; i < e_hi - e_lo; ++i) {
    const int e = fwd ? e_lo + i : e_hi - 1 - i;
    const T* re = rb + (long long)e * NK * nk;
    R ux = R(0), uy = R(0);
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      T rv = re[(long long)q * nk];
      if constexpr (RH) {
        rv.x *= sc;
        rv.y *= sc;
        rv = basis_round<RH>(rv);
      }
      ux += Dst[q] * rv.x;
      uy += Dst[q] * rv.y;
    }
    const R scm = RH ? R(1) : sc;   // RH: the scale is already in rv
    s.x = ux * scm * inv_qd + alpha * s.x;
    s.y = uy * scm * inv_qd + alpha * s.y;
    A *= alpha;
  }
  const long long m = ((long long)b * nchunk + c) * nk + j;
  mapA[m] = A;
  mapS[m] = s;
}

template <int NK, typename R, typename O = typename Cplx<R>::type>
__global__ void __launch_bounds__(32 * kChunksPerBlock) kline_apply_kernel(
    const typename Cplx<R>::type* __restrict__ r, typename Cplx<R>::type* __restrict__ z,
    __nv_bfloat162* __restrict__ zb, const R* __restrict__ kvec, const R* __restrict__ dinv,
    const R* __restrict__ hvec, const R* __restrict__ qd, const R* __restrict__ mapA,
    const typename Cplx<R>::type* __restrict__ mapS, int n_el, int nk, long long N, long long r_stride, int L,
    int nchunk, const int* __restrict__ mask, const R* __restrict__ rscale = nullptr,
    O* __restrict__ rout = nullptr, long long rout_stride = 0) {
  using T = typename Cplx<R>::type;
  constexpr bool RH = std::is_same<O, __half2>::value;
  const int j = blockIdx.x * 32 + threadIdx.x;
  const int c = blockIdx.y * kChunksPerBlock + threadIdx.y;
  const int b = blockIdx.z;
  if (j >= nk || c >= nchunk || (mask && !mask[b])) return;
  const long long bj = (long long)b * nk + j;
  const bool fwd = kvec[j] > R(0);
  const int st = fwd ? NK - 1 : 0;
  // incoming state: the maps of the chunks upwind of c, in sweep order
  T s;
  s.x = R(0);
  s.y = R(0);
  const long long mb = (long long)b * nchunk * nk + j;
  if (fwd) {
#pragma unroll 4
    for (int cc = 0; cc < c; ++cc) {
      const R a = mapA[mb + (long long)cc * nk];
      const T v = mapS[mb + (long long)cc * nk];
      s.x = a * s.x + v.x;
      s.y = a * s.y + v.y;
    }
  } else {
#pragma unroll 4
    for (int cc = nchunk - 1; cc > c; --cc) {
      const R a = mapA[mb + (long long)cc * nk];
      const T v = mapS[mb + (long long)cc * nk];
      s.x = a * s.x + v.x;
      s.y = a * s.y + v.y;
    }
  }
  R D[NK * NK], h[NK];
#pragma unroll
  for (int q = 0; q < NK * NK; ++q) D[q] = dinv[bj * NK * NK + q];
#pragma unroll
  for (int q = 0; q < NK; ++q) h[q] = hvec[bj * NK + q];
  const R inv_qd = qd[b] > R(0) ? rcp(qd[b]) : R(0);
  const R sc = rscale ? rscale[b] : R(1);
  const int e_lo = c * L, e_hi = min(n_el, e_lo + L);
  const T* rb = r + (long long)b * r_stride + j;
  T* zbase = z + (long long)b * N + j;
  O* obase = rout ? rout + (long long)b * rout_stride + j : nullptr;
  for (int i = 0; i < e_hi - e_lo; ++i) {
    const int e = fwd ? e_lo + i : e_hi - 1 - i;
    const T* re = rb + (long long)e * NK * nk;
    T rv[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      rv[q] = re[(long long)q * nk];
      if (rscale) {
        rv[q].x *= sc;
        rv[q].y *= sc;
      }
      rv[q] = basis_round<RH>(rv[q]);
      // the scaled input is the next Krylov basis vector: written here, so no separate pass
      if (obase) basis_store(obase[(long long)e * NK * nk + (long long)q * nk], rv[q]);
    }
    T snew = s;
#pragma unroll
    for (int a = 0; a < NK; ++a) {
      R ux = R(0), uy = R(0);
#pragma unroll
      for (int q = 0; q < NK; ++q) {
        ux += D[a * NK + q] * rv[q].x;
        uy += D[a * NK + q] * rv[q].y;
      }
      T zv;
      zv.x = ux * inv_qd - h[a] * s.x;
      zv.y = uy * inv_qd - h[a] * s.y;
      const long long o = (long long)e * NK * nk + (long long)a * nk;
      if (z) zbase[o] = zv;
      if (zb) zb[(long long)b * N + j + o] = __floats2bfloat162_rn((float)zv.x, (float)zv.y);
      if (a == st) snew = zv;
    }
    s = snew;
  }
}

// Maps, fold and sweep in one launch: thread (line jl, chunk c) of a block of KL lines and all nchunk chunks.  The loads
// of a thread's whole chunk are in flight together (the two-kernel form had one element's at a time, 1.4 TB/s in
// its second kernel, and read r twice): r once, z or its BF16 copy and the basis vector written.  FP32: bound by the loads
// that 1.7 waves of blocks keep in flight (63 MB in 18 us, 3.4 TB/s); FP64: by its pipe (55% busy) and the chain of a chunk.
// 16 problems of 240 elements, Nk = 256, nK = 4, FP16 basis: 32 -> 18 us; 4 of 180 elements, Nk = 512:
// 18.5 -> 10.7 us; FP64, 2 problems of 240 elements (FP64 pipe, 16 us of sums): 41 -> 31 us.
template <typename R, int NK> struct FusedLen {   // registers bound it: 32 complex FP32 values, 16 FP64
  static constexpr int value = (sizeof(R) == 8 ? 16 : 32) / NK;
};
template <typename R> constexpr int kFusedThreads = sizeof(R) == 8 ? 256 : 512;
template <typename T, bool RH> struct Held { using type = T; };
template <typename T> struct Held<T, true> { using type = __half2; };
__device__ __forceinline__ float2 held_get(__half2 v) { return __half22float2(v); }
__device__ __forceinline__ float2 held_get(float2 v) { return v; }
__device__ __forceinline__ double2 held_get(double2 v) { return v; }

template <int NK, typename R, typename O = typename Cplx<R>::type>
__global__ void __launch_bounds__(kFusedThreads<R>) kline_fused_kernel(
    const typename Cplx<R>::type* __restrict__ r, typename Cplx<R>::type* __restrict__ z,
    __nv_bfloat162* __restrict__ zb, const R* __restrict__ kvec, const R* __restrict__ dinv,
    const R* __restrict__ hvec, const R* __restrict__ qd, int n_el, int nk, long long N, long long r_stride, int L,
    int nchunk, int KL, const int* __restrict__ mask, const R* __restrict__ rscale, O* __restrict__ rout,
    long long rout_stride) {
  using T = typename Cplx<R>::type;
  constexpr bool RH = std::is_same<O, __half2>::value;
  constexpr int LM = FusedLen<R, NK>::value;
  extern __shared__ double kl_smem[];
  const int warps = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  T* mapS = reinterpret_cast<T*>(kl_smem);           // [warps][KL]
  R* mapA = reinterpret_cast<R*>(mapS + warps * KL);
  const int jl = threadIdx.x % KL, c = threadIdx.x / KL;
  const int j = blockIdx.x * KL + jl, b = blockIdx.y;
  if (mask && !mask[b]) return;   // uniform over the block
  const bool on = j < nk && c < nchunk;
  const long long bj = (long long)b * nk + (j < nk ? j : 0);
  const bool fwd = kvec[j < nk ? j : 0] > R(0);
  const int st = fwd ? NK - 1 : 0;
  const int e_lo = c * L, len = on ? min(n_el, e_lo + L) - e_lo : 0;
  const T* rb = r + (long long)b * r_stride + j;
  const long long row = (long long)NK * nk;
  auto elem = [&](int i) { return (long long)(fwd ? e_lo + i : e_lo + len - 1 - i) * row; };
  T raw[LM][NK];
#pragma unroll
  for (int i = 0; i < LM; ++i)
    if (i < len)
#pragma unroll
      for (int q = 0; q < NK; ++q) raw[i][q] = rb[elem(i) + (long long)q * nk];
  const R sc = rscale ? rscale[b] : R(1);
  const R inv_qd = qd[b] > R(0) ? rcp(qd[b]) : R(0);   // a problem without data stays zero
  R D[NK * NK], h[NK];
#pragma unroll
  for (int q = 0; q < NK * NK; ++q) D[q] = dinv[bj * NK * NK + q];
#pragma unroll
  for (int q = 0; q < NK; ++q) h[q] = hvec[bj * NK + q];
  R Dst[NK], alpha = fwd ? -h[NK - 1] : -h[0];
#pragma unroll
  for (int q = 0; q < NK; ++q) Dst[q] = fwd ? D[(NK - 1) * NK + q] : D[q];
  // the chunk's map s -> A s + S from a zero start
  typename Held<T, RH>::type rv[LM][NK];
  R A = R(1);
  T s;
  s.x = s.y = R(0);
#pragma unroll
  for (int i = 0; i < LM; ++i)
    if (i < len) {
      R ux = R(0), uy = R(0);
#pragma unroll
      for (int q = 0; q < NK; ++q) {
        T v = raw[i][q];
        v.x *= sc;
        v.y *= sc;
        if constexpr (RH) rv[i][q] = __floats2half2_rn(v.x, v.y);
        else rv[i][q] = v;
        v = held_get(rv[i][q]);
        ux += Dst[q] * v.x;
        uy += Dst[q] * v.y;
      }
      s.x = ux * inv_qd + alpha * s.x;
      s.y = uy * inv_qd + alpha * s.y;
      A *= alpha;
    }
  // maps of the warp's 32 / KL chunks scanned in sweep order (a fold over all upwind chunks costs FP64 118
  // dependent operations at 60 chunks, 7 of 34 us), the warps' own maps through shared memory
  const int W = 32 / KL, pos = fwd ? lane / KL : W - 1 - lane / KL, up = fwd ? -KL : KL;
  for (int d = 1; d < W; d *= 2) {
    const R pA = __shfl_sync(~0u, A, lane + d * up);
    const R px = __shfl_sync(~0u, s.x, lane + d * up), py = __shfl_sync(~0u, s.y, lane + d * up);
    if (pos >= d) {
      s.x += A * px;
      s.y += A * py;
      A *= pA;
    }
  }
  if (pos == W - 1) {
    mapA[warp * KL + jl] = A;
    mapS[warp * KL + jl] = s;
  }
  R exA = __shfl_sync(~0u, A, lane + up);
  T ex;
  ex.x = __shfl_sync(~0u, s.x, lane + up);
  ex.y = __shfl_sync(~0u, s.y, lane + up);
  // the scaled input is the next Krylov basis vector
  if (rout) {
    O* o = rout + (long long)b * rout_stride + j;
#pragma unroll
    for (int i = 0; i < LM; ++i)
      if (i < len)
#pragma unroll
        for (int q = 0; q < NK; ++q) o[elem(i) + (long long)q * nk] = rv[i][q];
  }
  __syncthreads();
  // incoming state: the maps of the upwind warps, then of the upwind chunks of this one
  s.x = s.y = R(0);
  const int first = fwd ? 0 : warps - 1, step = fwd ? 1 : -1, cnt = fwd ? warp : warps - 1 - warp;
  for (int i = 0; i < cnt; ++i) {
    const int m = (first + i * step) * KL + jl;
    s.x = mapA[m] * s.x + mapS[m].x;
    s.y = mapA[m] * s.y + mapS[m].y;
  }
  if (pos > 0) {
    s.x = exA * s.x + ex.x;
    s.y = exA * s.y + ex.y;
  }
  T* zo = z ? z + (long long)b * N + j : nullptr;
  __nv_bfloat162* zbo = zb ? zb + (long long)b * N + j : nullptr;
#pragma unroll
  for (int i = 0; i < LM; ++i)
    if (i < len) {
      const long long o = elem(i);
      T snew = s;
#pragma unroll
      for (int a = 0; a < NK; ++a) {
        R ux = R(0), uy = R(0);
#pragma unroll
        for (int q = 0; q < NK; ++q) {
          const T v = held_get(rv[i][q]);
          ux += D[a * NK + q] * v.x;
          uy += D[a * NK + q] * v.y;
        }
        T zv;
        zv.x = ux * inv_qd - h[a] * s.x;
        zv.y = uy * inv_qd - h[a] * s.y;
        if (zo) zo[o + (long long)a * nk] = zv;
        if (zbo) zbo[o + (long long)a * nk] = __floats2bfloat162_rn((float)zv.x, (float)zv.y);
        if (a == st) snew = zv;
      }
      s = snew;
    }
}

// Lines per block of the fused form: those that make 64-byte rows (with more, a block's 256 threads are reached at a few
// chunks, and a lone problem leaves SMs idle).  The scan's order follows from it, so it does not depend on the
// batch.  0 where the two-kernel form is taken (long chunks, or too many of them).
template <typename R, int NK>
inline int fused_lines(int n_el, int L) {
  constexpr int lines = 64 / (2 * (int)sizeof(R));
  return L > FusedLen<R, NK>::value || (n_el + L - 1) / L * lines > kFusedThreads<R> ? 0 : lines;
}

// Elements per chunk L.  The default: about 32 chunks per line (the incoming-state fold
// costs one map read per upwind chunk), at least 4 elements each; the autotuner times
// the candidates below and keeps the fastest per shape.  At most kMaxChunks chunks (the
// map buffers are sized for that).
constexpr int kMaxChunks = 64;
inline int chunk_len(int n_el) { return n_el / 32 > 4 ? (n_el + 31) / 32 : 4; }
inline int chunk_count_for(int n_el, int L) { return (n_el + L - 1) / L; }
inline int chunk_count(int n_el) { return chunk_count_for(n_el, chunk_len(n_el)); }
inline std::vector<int> chunk_len_candidates(int n_el) {
  std::vector<int> out;
  int last = -1;
  for (int L : {2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128}) {
    if (L > n_el && !out.empty()) break;
    const int nc = chunk_count_for(n_el, L);
    if (nc > kMaxChunks || nc == last) continue;
    out.push_back(L);
    last = nc;
  }
  if (out.empty()) out.push_back(chunk_len(n_el));
  return out;
}

}  // namespace kline
}  // namespace wg
