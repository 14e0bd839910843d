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
// the fraction.  The sum's low word holds the fraction's 32 bits, its high word
// the cell; a t outside [2^20, 2^21) has a high word that clamps to the same
// end of the line as c.
constexpr double DD_MAGIC = 1572864.0;  // 1.5 2^20
struct DdPos {
  int k;
  unsigned l;  // fraction x 2^32 (all ones: c >= N, a fraction of 1)
};
__device__ __forceinline__ DdPos dd_pos(double t, int N) {
  DdPos p{max(__double2hiint(t), 0x41300000) - 0x41380000, (unsigned)__double2loint(t)};
  if ((unsigned)p.k >= (unsigned)N) {
    p.l = p.k < 0 ? 0u : 0xffffffffu;
    p.k = p.k < 0 ? 0 : N - 1;
  }
  return p;
}
constexpr float DD_ULP = 2.3283064365386963e-10f;  // 2^-32
__device__ __forceinline__ void dd_cell(double t, int N, int& k, float& f) {
  const DdPos p = dd_pos(t, N);
  k = p.k;
  f = (float)p.l * DD_ULP;  // within 2^-25 of 1 it rounds to 1
}

// A centre position that FP32 offsets are added to, as t = c + DD_MAGIC24: its
// fraction's 24 bits, rounded (the offsets round at 2^-24 as well).
constexpr double DD_MAGIC24 = DD_MAGIC + 2.98023223876953125e-8;  // + 2^-25
__device__ __forceinline__ float dd_fraction24(double t) {
  return (float)((unsigned)__double2loint(t) >> 8) * 5.9604644775390625e-8f;
}

// The walk from p to e over a footprint of 1 / inv cells: w0 on the value at
// p.k, we on the value at e.k (0 when the cells are the same: it is the start
// value again), wm on the interior values between, if any.  Each is the part of
// the cell inside the footprint, over the footprint's length, so all are
// positive: up (inv > 0) 1 - f0 and f1, down f0 and 1 - f1, the same cell
// |f1 - f0|.  A part is taken as a whole number of 2^-32 cells and rounded to a
// float once: a ray that only grazes the masked image has a row sum of one or
// two small parts, and the residual is divided by it, so a part must be right
// relative to itself.  (With 24-bit fractions, and 1 - f in FP32, a row sum of
// 1e-4 pixels was 1e-4 off and some solves 1e-5; now 95 solves of 160^2 to
// 768^2 are within 1.8e-7.)
__device__ __forceinline__ void dd_walk(const DdPos& p, const DdPos& e, float inv, float& w0, float& wm, float& we) {
  const unsigned dn = (unsigned)(__float_as_int(inv) >> 31);  // all ones when down
  const unsigned a = p.l ^ ~dn, b = e.l ^ dn;
  const bool same = e.k == p.k;
  wm = fabsf(inv);
  const float s = wm * DD_ULP;
  w0 = (float)(same ? a + b + 1u : a) * s;
  we = (float)(same ? 0u : b) * s;
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
