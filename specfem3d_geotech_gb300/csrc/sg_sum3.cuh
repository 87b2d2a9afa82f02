// sg_sum3.cuh -- the dots and scalars of the FP32 PCG in FP32 instructions
// alone, with no fewer bits than FP64 keeps.
//
// An FP64 instruction holds the SM's FP64 unit for some 19 cycles a warp, and
// the FP64 trees over a block's warps and up to 32 sums took longer than the
// grid barrier of the persistent kernel.  A thread's products are exact (a*b =
// p + e with e = fma(a,b,-p)) and go into a two-float sum, in groups where a thread
// has many; from there on, over lanes, warps and blocks, a sum is three floats
// whose additions keep every rounding error but those of the third (T. J. Dekker,
// A floating-point technique for extending the available precision, Numer. Math.
// 18, 1971; D. E. Knuth's two-sum): some 70 bits of the sum of the absolute
// values.  Median relative error of a dot, a two-float sum per thread and an FP64
// tree against this: 1e-16, 1e-22 at 200 rows; 4e-16, 2e-16 at 120,000; 6e-16,
// 4e-16 at 1.6 million.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace sg {

// a product that is not contracted with the sum that takes it
__host__ __device__ __forceinline__ float mul_rn(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
// s = fl(a + b), and what that left out
__host__ __device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = a + b, bb = s - a;
  err = (a - (s - bb)) + (b - bb);
  return s;
}

struct Sum3 {
  float h, l, m;
  __host__ __device__ __forceinline__ void add(const Sum3& y) {
    float e, f, g;
    h = two_sum(h, y.h, e);
    const float s = two_sum(l, y.l, f);
    l = two_sum(s, e, g);
    m = (m + y.m) + (f + g);
  }
  __host__ __device__ __forceinline__ double value() const { return (double)h + ((double)l + (double)m); }
};
__host__ __device__ __forceinline__ Sum3 zero3() { return Sum3{0.f, 0.f, 0.f}; }
// An FP64 number as three floats, exactly while they are not subnormal
__host__ __device__ __forceinline__ Sum3 split3(double x) {
  const float h = (float)x;
  const double r = x - (double)h;
  const float l = (float)r;
  return Sum3{h, l, (float)(r - (double)l)};
}
// the same number with |l| at most half an ulp of h, and m of l
__host__ __device__ __forceinline__ Sum3 norm3(const Sum3& x) {
  float s, t;
  Sum3 y;
  s = two_sum(x.l, x.m, t);
  y.h = two_sum(x.h, s, s);
  y.l = two_sum(s, t, y.m);
  return y;
}
// a / b in FP32, a and b of norm3: the quotient of the high parts and two
// corrections by the remainder, rounded once
__host__ __device__ __forceinline__ float div3(const Sum3& a, const Sum3& b) {
  const float q0 = a.h / b.h, rb = 1.f / b.h;
  if (!(fabsf(q0) <= 3.4028234e38f)) return q0;   // no remainder to correct by
  // a - q0 b: the high parts' remainder is exact
  const float w = mul_rn(q0, b.l), we = fmaf(q0, b.l, -w);
  float t, e;
  const float r = two_sum(a.l, -w, t);
  const float dh = two_sum(fmaf(-q0, b.h, a.h), r, e);
  const float dl = e + ((t - we) + fmaf(-q0, b.m, a.m));
  const float q1 = mul_rn(dh, rb);
  const float q2 = mul_rn(fmaf(-q1, b.h, dh) + fmaf(-q1, b.l, dl), rb);
  const float s = q0 + q1;
  return s + ((q1 - (s - q0)) + q2);
}
// x <= y, of norm3
__host__ __device__ __forceinline__ bool at_most(const Sum3& x, const Sum3& y) {
  return (x.h - y.h) + ((x.l - y.l) + (x.m - y.m)) <= 0.f;
}

// Dot accumulator of one thread: exact products in a two-float sum.  Its error
// grows with the number of sums that lo has taken.
struct CompSum {
  float hi = 0.f, lo = 0.f;
  __host__ __device__ __forceinline__ void set(float a, float b) {   // the first product, exactly
    hi = mul_rn(a, b);
    lo = fmaf(a, b, -hi);
  }
  __host__ __device__ __forceinline__ void add(float a, float b) {
    const float p = mul_rn(a, b), e = fmaf(a, b, -p);
    float err;
    hi = two_sum(hi, p, err);
    lo += err + e;
  }
  __host__ __device__ __forceinline__ void add(const CompSum& x) {   // a group's sum
    float err;
    hi = two_sum(hi, x.hi, err);
    lo += err + x.lo;
  }
  __host__ __device__ __forceinline__ Sum3 sum() const { return Sum3{hi, lo, 0.f}; }
};
// the same for threads that add many products one by one: three floats
struct CompSum3 {
  float hi = 0.f, lo = 0.f, ll = 0.f;
  __host__ __device__ __forceinline__ void add(float a, float b) {
    const float p = mul_rn(a, b), e = fmaf(a, b, -p);
    float err, f, g;
    hi = two_sum(hi, p, err);
    const float s = two_sum(err, e, f);
    lo = two_sum(lo, s, g);
    ll += f + g;
  }
  __host__ __device__ __forceinline__ Sum3 sum() const { return Sum3{hi, lo, ll}; }
};

}  // namespace sg
