// Deterministic reductions.  FP64 arithmetic and FP64 conversions run at
// 1/64 of the FP32 rate on this GPU, so block-level sums of FP64 values are
// done in float-float (a hi/lo pair of FP32 numbers combined with
// error-free TwoSum, ~48 significant bits), entered and left by integer
// conversions, with one FP64 addition per value at the end.  The tree shape
// is fixed, so results are bitwise reproducible.
#pragma once
#include <cuda_runtime.h>

#include "softcvt.cuh"

namespace mdsc {

struct FF {
  float hi, lo;
};

// x as a float-float pair (48 bits), by integer instructions
__device__ __forceinline__ FF ff_from(double x) {
  FF r;
  soft_split(x, r.hi, r.lo);
  return r;
}

__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (b.hi - bb);
  const float lo = a.lo + b.lo + err;
  FF r;
  r.hi = s + lo;
  r.lo = lo - (r.hi - s);
  return r;
}

__device__ __forceinline__ FF ff_warp_sum(FF v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    FF o;
    o.hi = __shfl_xor_sync(0xffffffffu, v.hi, off);
    o.lo = __shfl_xor_sync(0xffffffffu, v.lo, off);
    v = ff_add(v, o);
  }
  return v;
}

// Sums NV float-float values over a block of NT threads (an FP32 value x
// enters as {x, 0}); thread 0 gets the totals in out[].  The warps' sums are
// added in float-float too, so each value costs one FP64 addition, at the
// end.  sh must hold NV * NT/32 doubles.
template <int NV, int NT>
__device__ __forceinline__ void block_sum(const FF (&v)[NV], double* sh, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FF* shf = reinterpret_cast<FF*>(sh);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    FF w = ff_warp_sum(v[c]);
    if (lane == 0) shf[c * (NT / 32) + warp] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      FF s = shf[c * (NT / 32)];
      for (int k = 1; k < NT / 32; ++k) s = ff_add(s, shf[c * (NT / 32) + k]);
      out[c] = soft_f2d(s.hi) + soft_f2d(s.lo);
    }
  }
  __syncthreads();
}

// Same, for FP64 values (split into float-float by integer instructions,
// 48 bits).
template <int NV, int NT>
__device__ __forceinline__ void block_sum(const double (&v)[NV], double* sh, double* out) {
  FF f[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) f[c] = ff_from(v[c]);
  block_sum<NV, NT>(f, sh, out);
}

__device__ __forceinline__ FF ff_of(float x) {
  FF r;
  r.hi = x;
  r.lo = 0.f;
  return r;
}

// NS sums of n floats `stride` apart, in order, in float-float (a dipole's
// real-space tile partials over its partner strips): hi + lo; the sums' floats
// are `next` apart.  W loads of each at a time; the ones past the end are zeros,
// which change nothing.
template <int W, int NS>
__device__ __forceinline__ void strip_sums(const float* v, int n, long long stride, int next, FF (&out)[NS]) {
  float hi[NS], lo[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) hi[c] = lo[c] = 0.f;
  for (int k = 0; k < n; k += W) {
    float x[W][NS];
#pragma unroll
    for (int q = 0; q < W; ++q)
#pragma unroll
      for (int c = 0; c < NS; ++c) x[q][c] = k + q < n ? v[(k + q) * stride + c * next] : 0.f;
#pragma unroll
    for (int q = 0; q < W; ++q)
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        const float sum = hi[c] + x[q][c];
        const float bb = sum - hi[c];
        lo[c] += (hi[c] - (sum - bb)) + (x[q][c] - bb);
        hi[c] = sum;
      }
  }
#pragma unroll
  for (int c = 0; c < NS; ++c) {
    out[c].hi = hi[c] + lo[c];
    out[c].lo = lo[c] - (out[c].hi - hi[c]);
  }
}

// m1 g2 - m2 g1, one component of a cross product with FP32 factors, high and
// low parts (the roundings written out: two kernels form it)
__device__ __forceinline__ FF ff_cross(float m1, FF g2, float m2, FF g1) {
  return FF{__fmaf_rn(m1, g2.hi, -__fmul_rn(m2, g1.hi)), __fmaf_rn(-m2, g1.lo, __fmul_rn(m1, g2.lo))};
}

// one Kahan addition: (fo, fc) += v
__device__ __forceinline__ void kahan(float& fo, float& fc, float v) {
  const float y = __fadd_rn(v, -fc);
  const float t = __fadd_rn(fo, y);
  fc = __fadd_rn(__fadd_rn(t, -fo), -y);
  fo = t;
}

// NS sums of n k tiles' sums `stride` apart in order, added in `parts` parts and
// the parts the same way: fo - fc; the sums' floats are `next` apart.  W loads of
// each at a time in flight.
template <int W, int NS>
__device__ __forceinline__ void ktile_sums(const float* in, int n, int stride, int next, int parts, FF (&out)[NS]) {
  const int per = parts == 1 ? n : (n + parts - 1) / parts;
  float po[NS], pc[NS], fo[NS], fc[NS], cs[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) po[c] = pc[c] = fo[c] = fc[c] = cs[c] = 0.f;
  auto close = [&] {  // a part ends
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      kahan(fo[c], fc[c], po[c]);
      cs[c] = __fadd_rn(cs[c], pc[c]);
      po[c] = pc[c] = 0.f;
    }
  };
  int in_part = 0, done = 0;
  for (int t0 = 0; t0 < n; t0 += W) {
    float v[W][NS];
#pragma unroll
    for (int q = 0; q < W; ++q)
#pragma unroll
      for (int c = 0; c < NS; ++c) v[q][c] = t0 + q < n ? in[(long long)(t0 + q) * stride + c * next] : 0.f;
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (t0 + q < n) {
#pragma unroll
        for (int c = 0; c < NS; ++c) kahan(po[c], pc[c], v[q][c]);
        if (parts > 1 && ++in_part == per) {
          close();
          in_part = 0;
          ++done;
        }
      }
  }
  if (parts > 1)
    for (; done < parts; ++done) close();  // the last part if it is not full, and empty ones
#pragma unroll
  for (int c = 0; c < NS; ++c) out[c] = parts == 1 ? FF{po[c], -pc[c]} : FF{fo[c], -__fadd_rn(fc[c], cs[c])};
}

}  // namespace mdsc
