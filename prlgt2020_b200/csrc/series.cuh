// series.cuh -- scalar parts of the truncated power series of 3x3 complex
// matrices (the reference's ptSU3, QCDpt.h:42-226): complex arithmetic, flags,
// twists, the float-float numbers of the compensated product.  The series
// themselves are in wseries.cuh.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nspt {

__device__ __forceinline__ double2 cz() { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.y * b.x + a.x * b.y);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double x) {
  return make_double2(a.x * x, a.y * x);
}
__device__ __forceinline__ bool cis0(double2 a) { return a.x == 0.0 && a.y == 0.0; }
// acc += a * b  (4 FP64 FMAs)
__device__ __forceinline__ void cfma(double2 &acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}
// flag of a product: a0*b0, or an exact 0 when both are 0 (QCDpt.h:102-104)
__device__ __forceinline__ double2 flag_mul(double2 a0, double2 b0) {
  return (cis0(a0) && cis0(b0)) ? cz() : cmul(a0, b0);
}

// Twist matrices Omega_d and Omega_d^dag (twistmatrices.h:158-240).
__constant__ double2 c_om[4][9];
__constant__ double2 c_omd[4][9];

// 3x3 complex product r = a * b, row major (SU3::operator*, MyMath.h:791-849).
__device__ __forceinline__ void m3_mul(double2 *r, const double2 *a, const double2 *b) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int q = 0; q < 3; q++) {
      double2 t = cmul(a[3 * i], b[q]);
      t = cadd(t, cmul(a[3 * i + 1], b[3 + q]));
      t = cadd(t, cmul(a[3 * i + 2], b[6 + q]));
      r[3 * i + q] = t;
    }
}

// Omega U Omega^dag for every twisted face a read crossed: backward wraps
// first (Omega_d^dag U Omega_d), then forward wraps, as the reference's
// backward copy slabs hold them (lattice.h:733-790, nspt.cc:221-253).
// m is row major.
__device__ __forceinline__ void twist3(double2 *m, unsigned tb, unsigned tf) {
  double2 t[9];
#pragma unroll
  for (int d = 1; d < 4; d++)
    if ((tb >> d) & 1) {
      m3_mul(t, c_omd[d], m);
      m3_mul(m, t, c_om[d]);
    }
#pragma unroll
  for (int d = 1; d < 4; d++)
    if ((tf >> d) & 1) {
      m3_mul(t, c_om[d], m);
      m3_mul(m, t, c_omd[d]);
    }
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// ---------------- compensated float-float Cauchy product ----------------
//
// The truncated product with every multiply-add of the triangle in float-float
// arithmetic: a double x is split into
// hi = fl32(x 2^e) and lo = fl32(x 2^e - hi) (48 significant bits together);
// a product of two such numbers is formed with an exact FP32 product
// (p = xh yh, err = fma(xh, yh, -p)) plus the cross terms, and added to the
// accumulator by an error-free two-sum whose error is carried in the low
// word.  Order i of the left operand and order j of the right one are
// scaled by 2^(e i) and 2^(e j) before the split (exact), so that orders of
// very different size keep inside the FP32 exponent range; the order-k
// result is scaled back by 2^(-e k) when it is rejoined into FP64.  The flag
// terms, the output and everything around the products stay FP64.
struct ffc {
  float rh, rl, ih, il;  // re = rh + rl, im = ih + il
};

// 2^n as a double, exact for -1022 <= n <= 1023
__device__ __forceinline__ double pow2i(int n) { return __hiloint2double((1023 + n) << 20, 0); }

__device__ __forceinline__ ffc ff_split(double2 v, double scale) {
  const double x = v.x * scale, y = v.y * scale;
  const float xh = __double2float_rn(x), yh = __double2float_rn(y);
  return {xh, __double2float_rn(x - (double)xh), yh, __double2float_rn(y - (double)yh)};
}

// (ah, al) += (xh, xl) (yh, yl); rounding-explicit so nothing is contracted
__device__ __forceinline__ void ff_mac(float &ah, float &al, float xh, float xl, float yh,
                                       float yl) {
  const float p = __fmul_rn(xh, yh);
  float e = __fmaf_rn(xh, yh, -p);
  e = __fmaf_rn(xh, yl, e);
  e = __fmaf_rn(xl, yh, e);
  const float s = __fadd_rn(ah, p);
  const float b = __fsub_rn(s, ah);
  const float err = __fadd_rn(__fsub_rn(ah, __fsub_rn(s, b)), __fsub_rn(p, b));
  ah = s;
  al = __fadd_rn(al, __fadd_rn(err, e));
}

__device__ __forceinline__ void ff_cmac(ffc &acc, const ffc &a, const ffc &b) {
  ff_mac(acc.rh, acc.rl, a.rh, a.rl, b.rh, b.rl);
  ff_mac(acc.rh, acc.rl, -a.ih, -a.il, b.ih, b.il);
  ff_mac(acc.ih, acc.il, a.rh, a.rl, b.ih, b.il);
  ff_mac(acc.ih, acc.il, a.ih, a.il, b.rh, b.rl);
}

__device__ __forceinline__ double inv_factorial(int n) {
  double f = 1.0;
  for (int m = 2; m <= n; m++) f *= (double)m;
  return 1.0 / f;
}

}  // namespace nspt
