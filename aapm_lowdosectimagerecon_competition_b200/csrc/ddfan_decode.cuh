// ddfan_decode.cuh -- the position arithmetic shared by the table-free kernels
// and the slice-major REF backprojector.
#pragma once
#include <cuda_runtime.h>

namespace ddfan {

// ============================================================ decode arithmetic
//
// A warp decodes 32 positions at a time for its gathers, so with few slices
// the decode is most of the work.  It keeps the FP64 formulas but none of
// FP64's slow companions: comparisons, divisions and conversions (which share
// a 4-lane unit) are replaced as below.

// Position c, as t = c + DD_MAGIC: the cell (clamped so that 0 <= c <= N) and
// the fraction.  The sum's low word holds 32 fraction bits, of which 24 are
// kept (DD_MAGIC's 2^-25 rounds them), its high word the cell; a t outside
// [2^20, 2^21) has a high word that clamps to the same end of the line as c.
constexpr double DD_MAGIC = 1572864.0 + 2.98023223876953125e-8;
__device__ __forceinline__ void dd_cell(double t, int N, int& k, float& f) {
  k = max(__double2hiint(t), 0x41300000) - 0x41380000;
  f = (float)((unsigned)__double2loint(t) >> 8) * 5.9604644775390625e-8f;
  if ((unsigned)k >= (unsigned)N) {
    f = k < 0 ? 0.f : 1.f;
    k = k < 0 ? 0 : N - 1;
  }
}

// The approximate reciprocal (relative error below 2^-22), and 1 / x within an
// ulp: one Newton step on it
__device__ __forceinline__ float dd_rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float dd_rcpf(float x) {
  const float r = dd_rcp_approx(x);
  return fmaf(r, fmaf(-x, r, 1.f), r);
}

// l = sqrt(l2) and 1 / l, for normal l2: the approximate reciprocal square root
// and one Newton step.  The step is added as a correction: as the factor
// 1.5 - l2 r r / 2, which rounds near 1, it would leave the approximation's bias
// in the result, and every sample of a voxel has the same one.
__device__ __forceinline__ void dd_length(float l2, float& l, float& rl) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l2));
  const float h = l2 * r, e = 0.5f * fmaf(-h, r, 1.f);
  rl = fmaf(r, e, r);
  l = fmaf(h, e, h);
}

// x as a double, exactly, for normal x, with integer instructions
__device__ __forceinline__ double dd_widen(float x) {
  const unsigned u = __float_as_uint(x);
  return __hiloint2double((int)(((u & 0x7fffffffu) >> 3) + 0x38000000u | (u & 0x80000000u)), (int)(u << 29));
}

// 1 / x in FP64 from a float seed within 2^-20: one Newton step (2^-40)
__device__ __forceinline__ double dd_newton(double x, float seed) {
  const double y = dd_widen(seed);
  return fma(y, fma(-x, y, 1.0), y);
}

// A voxel's ray from the source, for the decode: the vector (FP64, FP32)
struct DdRay {
  double x, y;
  float xf, yf;
};

// asin(cr / hypot(cr, dt)), the angle of a voxel's ray v from the central ray
// (cross and dot product of -s and v).  In front of the source (dt > 0) it is
// atan(cr / dt): with T = j / 64 the grid tangent nearest to cr / dt,
// atan(cr / dt) = atan(T) + atan(z), z = (cr - T dt) / (dt + T cr), |z| <=
// 1 / 128: z in FP64 and its Taylor series' next two terms, at most 1.6e-7, in
// FP32.  tab: (T, atan(T) of the library function); rays beyond 45 degrees
// call asin.
constexpr int DD_ATAN_N = 64;
__device__ __forceinline__ double2 dd_atan_entry(int j) {  // entry j of 0 .. 2 DD_ATAN_N
  const double t = (double)(j - DD_ATAN_N) / (double)DD_ATAN_N;
  return make_double2(t, atan(t));
}
__device__ __forceinline__ double dd_angle(const DdRay& v, double sx, double sy, float sxf, float syf, const double2* tab) {
  const double cr = fma(sy, v.x, -sx * v.y), dt = -fma(sx, v.x, sy * v.y);
  const float crf = fmaf(syf, v.xf, -sxf * v.yf), dtf = -fmaf(sxf, v.xf, syf * v.yf);
  const float tf = crf * dd_rcp_approx(dtf);
  if (!(dtf > 0.f && fabsf(tf) <= 1.f)) return asin(cr / sqrt(cr * cr + dt * dt));
  const float jf = fmaf(tf, (float)DD_ATAN_N, 12582912.f);  // 1.5 2^23: rounds to an integer
  const double2 q = tab[__float_as_int(jf) - 0x4b400000 + DD_ATAN_N];
  const float Tf = (jf - 12582912.f) * (1.f / (float)DD_ATAN_N);
  const float rf = dd_rcp_approx(fmaf(Tf, crf, dtf));
  const double z = fma(-q.x, dt, cr) * dd_newton(fma(q.x, cr, dt), rf);
  const float zf = fmaf(-Tf, dtf, crf) * rf, z2 = zf * zf;
  return fma(-z, dd_widen(z2 * fmaf(z2, -0.2f, 1.f / 3.f)), z) + q.y;
}

}  // namespace ddfan
