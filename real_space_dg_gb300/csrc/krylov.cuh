// Pieces of the Krylov solver (gmres.cu): basis loads, block reductions, the Givens step and the back substitution.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

namespace wg {
namespace {

constexpr int kMaxRestart = 256;   // Krylov length bound of the device Givens / staging buffers

// Basis loads of the FP32 inner solve: four consecutive complex values (32 bytes of an FP32 basis,
// 16 bytes of an FP16 one; N is a multiple of 4 there) as they come, and their value as floats.
template <typename VB> struct Quad;
template <> struct Quad<float2> {
  float4 u, v;
  __device__ __forceinline__ void load(const float2* p, long long n4) {
    u = __ldg(reinterpret_cast<const float4*>(p) + 2 * n4);
    v = __ldg(reinterpret_cast<const float4*>(p) + 2 * n4 + 1);
  }
  __device__ __forceinline__ void zero() { u = v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ float2 get(int i) const {
    return i == 0 ? make_float2(u.x, u.y) : i == 1 ? make_float2(u.z, u.w)
                                                   : i == 2 ? make_float2(v.x, v.y) : make_float2(v.z, v.w);
  }
};
template <> struct Quad<__half2> {
  uint4 u;
  __device__ __forceinline__ void load(const __half2* p, long long n4) {
    u = __ldg(reinterpret_cast<const uint4*>(p) + n4);
  }
  __device__ __forceinline__ void zero() { u = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ float2 get(int i) const {
    const unsigned w = i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w;
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
};
__device__ __forceinline__ float2 ld_one(const float2& v) { return v; }
__device__ __forceinline__ double2 ld_one(const double2& v) { return v; }
__device__ __forceinline__ float2 ld_one(const __half2& v) { return __half22float2(v); }

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Complex multiply-subtract in the vector's own precision: w -= v h.
__device__ __forceinline__ void cms(double2& w, const double2& v, const double2& h) {
  w.x = fma(-v.x, h.x, fma(v.y, h.y, w.x));
  w.y = fma(-v.x, h.y, fma(-v.y, h.x, w.y));
}
__device__ __forceinline__ void cms(float2& w, const float2& v, const float2& h) {
  w.x = fmaf(-v.x, h.x, fmaf(v.y, h.y, w.x));
  w.y = fmaf(-v.x, h.y, fmaf(-v.y, h.x, w.y));
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over a block of up to 256 threads; the result is valid in warp 0.
__device__ double block_sum1(double v) {
  __shared__ double s[8];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  if (lane == 0) s[w] = v;
  __syncthreads();
  double r = 0;
  if (threadIdx.x < 32) {
    r = lane < nw ? s[lane] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

// The last block of a problem to finish a grid-wide pass (per-problem ticket
// counter; the threadFenceReduction pattern: every block fences its partial
// results, takes a ticket, and the block holding the last ticket reduces them and
// resets the counter for the next launch on the stream).  No block waits.
__device__ __forceinline__ bool last_block_of_problem(int* __restrict__ count, int b) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&count[b], 1) == (int)(gridDim.x * gridDim.z) - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Givens step k of problem b (one warp): rotate the new Hessenberg column by the
// previous rotations, make the next rotation, update g and deactivate the problem
// once the residual estimate |g[k+1]| reaches its target.  H is column-major per
// problem (H[b][col*(m+1)+row]), cs/sn/g per problem; h_next = H[k+1][k].
// Rotation i maps (t_i, h_{i+1}) to (r_i, t_{i+1}) with r_i = c t + s h and t_{i+1} = -conj(s) t + conj(c) h:
// t is a first-order recurrence, so a warp scan of its affine maps (|factor| <= 1) gives 32 rotations in
// about 55 FP64 instructions instead of 14 per rotation in sequence (each takes a quarter's FP64 pipe for
// 64 cycles whatever the number of lanes).  This tail runs after the last block of an update, so it is on
// the critical path of every Arnoldi step: the update launches of a 1,152-unknown solve (k up to 50)
// took 28.1 us on average with the sequential rotations, 21.5 us with the scan.
__device__ void givens_warp(double2* __restrict__ H, double2* __restrict__ cs, double2* __restrict__ sn,
                            double2* __restrict__ g, int* __restrict__ active, int* __restrict__ kused,
                            const double* __restrict__ target, int b, int k, int pstride, int m, double h_next) {
  const int lane = threadIdx.x & 31;
  double2* col = H + (long long)b * pstride * m + (long long)k * pstride;
  double2* c = cs + b * m;
  double2* s = sn + b * m;
  double2* gg = g + b * pstride;
  const double2 gk = gg[k];
  const double tg = target[b];
  double2 t = col[0];
  for (int i0 = 0; i0 < k; i0 += 32) {
    const int i = i0 + lane;
    const bool in = i < k;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 ci = in ? c[i] : zero, si = in ? s[i] : zero, hn = in ? col[i + 1] : zero;
    double2 A = in ? make_double2(-si.x, si.y) : make_double2(1.0, 0.0);
    double2 Bv = make_double2(fma(ci.x, hn.x, ci.y * hn.y), fma(ci.x, hn.y, -ci.y * hn.x));
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      double2 Ap, Bp;
      Ap.x = __shfl_up_sync(0xffffffffu, A.x, o);
      Ap.y = __shfl_up_sync(0xffffffffu, A.y, o);
      Bp.x = __shfl_up_sync(0xffffffffu, Bv.x, o);
      Bp.y = __shfl_up_sync(0xffffffffu, Bv.y, o);
      if (lane >= o) {
        Bv = make_double2(fma(A.x, Bp.x, fma(-A.y, Bp.y, Bv.x)), fma(A.x, Bp.y, fma(A.y, Bp.x, Bv.y)));
        A = make_double2(fma(A.x, Ap.x, -A.y * Ap.y), fma(A.x, Ap.y, A.y * Ap.x));
      }
    }
    const double2 tn = make_double2(fma(A.x, t.x, fma(-A.y, t.y, Bv.x)), fma(A.x, t.y, fma(A.y, t.x, Bv.y)));
    double2 ti;   // t_i: the previous lane's t_{i+1}
    ti.x = __shfl_up_sync(0xffffffffu, tn.x, 1);
    ti.y = __shfl_up_sync(0xffffffffu, tn.y, 1);
    if (lane == 0) ti = t;
    if (in)
      col[i] = make_double2(fma(ci.x, ti.x, fma(-ci.y, ti.y, fma(si.x, hn.x, -si.y * hn.y))),
                            fma(ci.x, ti.y, fma(ci.y, ti.x, fma(si.x, hn.y, si.y * hn.x))));
    t.x = __shfl_sync(0xffffffffu, tn.x, 31);
    t.y = __shfl_sync(0xffffffffu, tn.y, 31);
  }
  const double d2 = fma(t.x, t.x, fma(t.y, t.y, h_next * h_next));
  double2 cc = make_double2(1.0, 0.0);
  double ss = 0.0, den = 0.0;
  if (d2 > 0.0) {
    const double inv = rsqrt(d2);
    den = d2 * inv;
    cc = make_double2(t.x * inv, -t.y * inv);
    ss = h_next * inv;
  } else if (d2 != 0.0) {   // NaN: passed on, the problem stops below
    den = d2;
    cc = make_double2(d2, d2);
    ss = d2;
  }
  const double2 gn = make_double2(-ss * gk.x, -ss * gk.y);
  if (lane == 0) {
    c[k] = cc;
    s[k] = make_double2(ss, 0.0);
    col[k] = make_double2(den, 0.0);
    col[k + 1] = make_double2(0.0, 0.0);
    gg[k + 1] = gn;
    gg[k] = make_double2(fma(cc.x, gk.x, -cc.y * gk.y), fma(cc.x, gk.y, cc.y * gk.x));
    kused[b] = k + 1;
    const double res2 = fma(gn.x, gn.x, gn.y * gn.y);
    if (!(res2 > tg * tg) || h_next == 0.0 || !isfinite(res2)) active[b] = 0;
  }
}

// y = R^-1 g for the rotated Hessenberg matrix R (upper triangular, column-major per
// problem), one warp per problem: column-oriented back substitution, the lanes update
// the remaining right-hand side with column i of R.  The inverse diagonal is formed for
// all rows at once first, and column i - 1 is loaded into registers while column i is
// applied, so the serial sweep waits on neither a division nor a load per row.
__global__ void backsolve_kernel(const double2* __restrict__ H, const double2* __restrict__ g,
                                 double2* __restrict__ y, float2* __restrict__ y32, const int* __restrict__ kused,
                                 int pstride, int m, int batch) {
  constexpr int JT = kMaxRestart / 32;   // column entries per lane
  __shared__ double2 acc[kMaxRestart + 1];
  __shared__ double2 dinv[kMaxRestart];
  const int b = blockIdx.x;
  const int lane = threadIdx.x;
  if (b >= batch) return;
  const int kk = kused[b];
  const double2* Hb = H + (long long)b * pstride * m;
  double2* yb = y + b * m;
  for (int i = lane; i < m; i += 32) {
    acc[i] = i < kk ? g[b * pstride + i] : make_double2(0, 0);
    if (i >= kk) yb[i] = make_double2(0, 0);
  }
  for (int i = lane; i < kk; i += 32) {
    const double2 d = Hb[(long long)i * pstride + i];
    const double dd = d.x * d.x + d.y * d.y;
    dinv[i] = dd > 0 ? make_double2(d.x / dd, -d.y / dd) : make_double2(0, 0);
  }
  double2 cur[JT], nxt[JT];
#pragma unroll
  for (int t = 0; t < JT; ++t) {
    const int j = lane + 32 * t;
    cur[t] = (kk > 0 && j < kk - 1) ? Hb[(long long)(kk - 1) * pstride + j] : make_double2(0, 0);
  }
  __syncwarp();
  for (int i = kk - 1; i >= 0; --i) {
#pragma unroll
    for (int t = 0; t < JT; ++t) {
      const int j = lane + 32 * t;
      nxt[t] = (i > 0 && j < i - 1) ? Hb[(long long)(i - 1) * pstride + j] : make_double2(0, 0);
    }
    const double2 yi = cmul(acc[i], dinv[i]);
    if (lane == 0) yb[i] = yi;
#pragma unroll
    for (int t = 0; t < JT; ++t) {
      const int j = lane + 32 * t;
      if (j < i) {
        const double2 u = cmul(cur[t], yi);
        acc[j].x -= u.x;
        acc[j].y -= u.y;
      }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < JT; ++t) cur[t] = nxt[t];
  }
  __syncwarp();
  if (y32)
    for (int i = lane; i < m; i += 32) {
      const double2 v = i < kk ? yb[i] : make_double2(0, 0);
      y32[b * m + i] = make_float2((float)v.x, (float)v.y);
    }
}

// Groups of four elements per block of the FP32 Gram-Schmidt kernels, a rule on the size of one problem alone: a problem's
// sums, and with them its bits, do not depend on the batch it is in.  Pieces of 4,096 and 2,048 elements against
// one wave of blocks for the batch, whole solves: 8 problems of 153,600 unknowns 26.7 and 26.6 ms, 16 of 245,760 63.4
// and 64.0, eight concurrent handles of 2 such 211 and 204, 4 of 368,640 67.9 and 67.5.  Half of both: 27.1, 64.0, 206, 69.3.
inline int dot_quads(long long N) { return N >= 1 << 17 ? 1024 : 512; }
inline int update_quads(long long N) { return N >= 1 << 17 ? 512 : N >= 1 << 16 ? 256 : 128; }

}  // namespace
}  // namespace wg
