// ddfan_dd_kernels.cuh -- projector kernels that read the values themselves
// instead of prefix-sum tables (DDFAN_SAT_DIRECT).
//
// Every sample of the branchless DD path is a difference of two linearly
// interpolated prefix sums, Phi(c1) - Phi(c0), with Phi(c) = S[k] + f v[k]
// (k = floor of the clamped c, f its fraction; AAPM_script/
// MultiSlicesProjGPU.cu:161-170, MultiSlicesBackGPU.cu:175-179).  The
// difference telescopes to the values between the two positions:
//   k1 == k0:  (f1 - f0) v[k0]
//   k1 >  k0:  (1 - f0) v[k0] + sum_{k0<k<k1} v[k] + f1 v[k1]
//   k1 <  k0:  -f0 v[k0] - sum_{k1<k<k0} v[k] + (f1 - 1) v[k1]
// -- the same number in exact arithmetic, with no cancellation in FP32 and
// without building or reading a table.  A DD footprint covers one to three
// values at the geometries this path serves (the axis is chosen so that a ray
// crosses at most one cell per line, and channel and pixel pitch are
// comparable), so a sample reads one float per slice plus the one it shares
// with its neighbour, where a 48-byte hi/lo cell read 12 bytes per slice per
// boundary.  Wider footprints walk more values (any width is correct).
//
// Layouts: the image [YN][XN][slices] and the sinogram operands
// [slot][U + 1][slices], slices padded to a multiple of 4 or 8 and read in
// vectors of that many; the image masked beforehand, the (weighted) residual
// with a zero guard channel U, so a walk that ends on the last boundary
// (index U, fraction 0) reads a zero.
#pragma once
#include <type_traits>

#include "ddfan_decode.cuh"
#include "ddfan_proj_kernels.cuh"

namespace ddfan {

// Resident CTAs per SM the register allocation is sized for (256 threads:
// 3 -> up to 80 registers, 2 -> 128).  Build-time knobs for tuning sweeps, like the tile shapes below.
#ifndef DDFAN_DD_FWD_MIN_CTAS
#define DDFAN_DD_FWD_MIN_CTAS 3
#endif
#ifndef DDFAN_DD_BACK_MIN_CTAS
#define DDFAN_DD_BACK_MIN_CTAS 2
#endif
// ============================================================ vectors of slices

// The slices a thread owns, loaded at once: 8 (32 bytes, one 256-bit load --
// half the load instructions and address arithmetic of two 128-bit ones), 4
// (16 bytes) or 1.  8 and 4 are kept as pairs for fma.rn.f32x2.
using u64 = unsigned long long;

template <int SV> struct Vec {
  static constexpr int Q = SV / 2;
  u64 q[Q];
};
template <> struct Vec<1> {
  float f;
};

__device__ __forceinline__ void vload(Vec<8>& v, const char* p) {
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
      : "=l"(v.q[0]), "=l"(v.q[1]), "=l"(v.q[2]), "=l"(v.q[3])
      : "l"(p));
}
__device__ __forceinline__ void vload(Vec<4>& v, const char* p) {
  asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(v.q[0]), "=l"(v.q[1]) : "l"(p));
}
__device__ __forceinline__ void vload(Vec<1>& v, const char* p) { v.f = __ldg(reinterpret_cast<const float*>(p)); }

constexpr unsigned DD_INNER = 0x80000000u;  // the walk has an interior value (offsets stay below 2^31 vectors)

// w in both halves of a 64-bit word
__device__ __forceinline__ u64 dup2(float w) {
  u64 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(w));
  return r;
}
__device__ __forceinline__ float lo2(u64 w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ float hi2(u64 w) { return __uint_as_float((unsigned)(w >> 32)); }

// a += w v (w in both halves of ww)
template <int SV>
__device__ __forceinline__ void vfma(Vec<SV>& a, u64 ww, const Vec<SV>& v) {
#pragma unroll
  for (int i = 0; i < Vec<SV>::Q; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a.q[i]) : "l"(ww), "l"(v.q[i]));
}
__device__ __forceinline__ void vfma(Vec<1>& a, u64 ww, const Vec<1>& v) { a.f = fmaf(lo2(ww), v.f, a.f); }

template <int SV>
__device__ __forceinline__ void vzero(Vec<SV>& a) {
#pragma unroll
  for (int i = 0; i < Vec<SV>::Q; ++i) a.q[i] = 0ull;
}
__device__ __forceinline__ void vzero(Vec<1>& a) { a.f = 0.f; }

template <int SV>
__device__ __forceinline__ float vget(const Vec<SV>& a, int s) {
  return (s & 1) ? hi2(a.q[s >> 1]) : lo2(a.q[s >> 1]);
}
__device__ __forceinline__ float vget(const Vec<1>& a, int) { return a.f; }

// ============================================================ forward projector

struct DdFwdArgs {
  const float* img;    // masked image [YN][XN][ZP vectors of SV slices]
  const float* imgT;   // its columns [XN][YN][ZP vectors] or null (fwd_thin_body)
  int ZP;
  const ViewGeom* vg;
  const double2* fc;   // [PN][U+1] boundary lines
  const float* cvd;    // [PN][U] 1 / |dir.axis|
  const int* order;    // CTA row -> view, x-major first (null = identity)
  float* out;          // [slot][orow][ostride]
  int orow, ostride;
  int PN, U, XN, YN;
  float dx;
  int zlo, zhi;        // slices written
  int sv;              // slices per thread (the kernel's SV)
  int zl;              // lanes of a channel group: vectors of a z-tile
  int vb0, nvb, nzt;   // first vector and vectors of [zlo, zhi); z-tiles of zl vectors
  int nseg;            // line segments a warp's lines are split into (1, 2, 4 or 8)
  int thin;            // few slices: fwd_thin_body (zl = 1)
  // fused OS-SART residual (AAPM_script/OSSART_AAPM.m:86-88); y null = plain projection
  const float* y;      // measured [views][U][ystride]
  const int* yview;    // slot -> measured view
  const float* rowsum; // [slot][U]
  const float* wgt;    // [slot][U] weight of the exact adjoint, or null
  int ystride;
};

// channels per thread of the forward projector (at most 3: s_m's layout)
#ifndef DDFAN_DD_FWD_CG
#define DDFAN_DD_FWD_CG 2
#endif

template <int SV>
struct DdFwdTile {
  static constexpr int NT = 256, NW = NT / 32;
  static constexpr int CG = DDFAN_DD_FWD_CG;
  static constexpr int REC = 128;      // (line, channel) walks a warp decodes at a time
  static constexpr int FLUSH = 32;     // lines per FP32 partial sum
  static constexpr int THIN_CG = 2;    // channels per thread of fwd_thin_body
  // dynamic shared memory of the ray totals, of either body
  static constexpr int DYN = (CG > THIN_CG ? CG : THIN_CG) * SV * NT * (int)sizeof(float);
};

// The lines that any footprint of channels [wc0, wc0 + n) meets, and of those
// the warp's segment.
__device__ __forceinline__ void dd_warp_lines(const double2* fcp, int wc0, int n, int U, double N, int nl, int seg,
                                              int nseg, int& lo, int& hi) {
  lo = hi = 0;
  if (wc0 >= U) return;
  int pl = nl, ph = 0, ql = nl, qh = 0;
  for (int b = threadIdx.x & 31; b <= n; b += 32) {
    const double2 f = __ldg(fcp + min(wc0 + b, U));
    int b0, b1, b2, b3;
    line_range(f.x, f.y, N, nl, b0, b1, b2, b3);
    pl = min(pl, b0);
    ph = max(ph, b1);
    ql = min(ql, b2);
    qh = max(qh, b3);
  }
  pl = __reduce_min_sync(0xffffffffu, pl);
  ph = __reduce_max_sync(0xffffffffu, ph);
  ql = __reduce_min_sync(0xffffffffu, ql);
  qh = __reduce_max_sync(0xffffffffu, qh);
  const int l0 = max(pl, ql), m = max(0, min(ph, qh) - l0);
  lo = l0 + m * seg / nseg;
  hi = l0 + m * (seg + 1) / nseg;
}

// Stores channel u of view p: the ray sums of slices [vb SV, vb SV + SV), or
// the OS-SART residual made of them.
template <int SV>
__device__ __forceinline__ void dd_fwd_store(const DdFwdArgs& a, int p, int u, int vb, float (&val)[SV]) {
  const size_t e = (size_t)p * a.U + u;
  const float cv = __ldg(a.cvd + e) * a.dx;
  float* oz = a.out + ((size_t)p * a.orow + u) * a.ostride + vb * SV;
  const float* yv = nullptr;
  float rs = 0.f, wt = 1.f;
  if (a.y) {
    rs = __ldg(a.rowsum + e);
    if (a.wgt) wt = __ldg(a.wgt + e);
    yv = a.y + ((size_t)__ldg(a.yview + p) * a.U + u) * a.ystride;
  }
#pragma unroll
  for (int s = 0; s < SV; ++s) {
    val[s] *= cv;
    const int zs = vb * SV + s;
    if (yv && zs >= a.zlo && zs < a.zhi) {
      // (y - A x) / rowSum where rowSum != 0, else A x (AAPM_script/OSSART_AAPM.m:88)
      val[s] = rs != 0.f ? __fdiv_rn(__fsub_rn(__ldg(yv + zs), val[s]), rs) : val[s];
      val[s] *= wt;
    }
  }
  if (SV >= 4 && (a.ostride & 3) == 0 && vb * SV >= a.zlo && vb * SV + SV <= a.zhi &&
      (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
#pragma unroll
    for (int s = 0; s + 4 <= SV; s += 4)
      *reinterpret_cast<float4*>(oz + s) = make_float4(val[s], val[s + 1], val[s + 2], val[s + 3]);
  } else {
#pragma unroll
    for (int s = 0; s < SV; ++s)
      if (vb * SV + s >= a.zlo && vb * SV + s < a.zhi) oz[s] = val[s];
  }
}

// What bounds it (c3 subset, 96 views x 736 channels x 512^2 x 128): the loads'
// latency, and behind it the L1 pipe -- 1.26 ms (1.29 in one tile of 128
// slices), of which 1.0 ms remain when every load hits L1; 14.2 GB cross from
// L2 (every view reads the image once: 12.9 GB) at 11 TB/s; 60 % of L1's
// wavefronts, 95 % L2 hits.  24 warps an SM at 80 registers and 2 channels a
// thread beat 16 warps at 128 with 3 channels (1.34 ms) or 2 (1.41).  Before: 1.90 ms (4 z-tiles of 4 slices a
// thread, no lines skipped).
//
// Warp = one view x (32 / zl) groups of CG consecutive channels x zl vectors
// of SV slices; CTA = 8 warps, on consecutive channels (and, when nseg > 1, on
// nseg segments of the lines, added up in shared memory at the end).  A
// thread walks its channels' footprints along each line: the value at the
// boundary two channels share is loaded once, so a line costs CG + 1 loads
// plus one for every footprint with an interior value, all issued before the
// first is used.  Every warp decodes its own walks (REC at a time, FP64
// boundary lines: each channel's two cell offsets and walk weights over
// 1 / footprint length, MultiSlicesProjGPU.cu:166-170) and synchronises with
// itself only.  Lines on which none of the warp's footprints meet the image
// are skipped (their weights are zero): a third of all (channel, line) pairs
// at the c2 geometry, whose detector covers more than the image.
template <int SV>
__device__ __forceinline__ void fwd_dd_body(const DdFwdArgs& a, int row, int cblk, int ztile) {
  using T = DdFwdTile<SV>;
  constexpr int NW = T::NW, CG = T::CG, REC = T::REC, VB = SV * 4;
  static_assert(CG >= 1 && CG <= 3, "s_m holds a start and three interior offsets");
  __shared__ float4 s_w[NW][REC];         // (w0, wm, we) / length, end offset (bits) of walk (line, group, j)
  __shared__ uint4 s_m[NW][REC / CG];     // (line, group): start offset, then each channel's interior one
  extern __shared__ float s_tot[];          // [CG * SV][NT]: this thread's totals at tid
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int ZL = a.zl, GW = 32 / ZL, CWW = GW * CG, CC = REC / CWW;
  const int g = lane / ZL, zi = lane - g * ZL;
  const int nseg = a.nseg, wch = w / nseg, seg = w - wch * nseg;
  const int wc0 = (cblk * (NW / nseg) + wch) * CWW;  // the warp's first channel
  const int p = a.order ? a.order[row] : row;
  const bool active = g < GW && ztile * ZL + zi < a.nvb && wc0 + g * CG < a.U;
  const int vb = a.vb0 + ztile * ZL + zi;
  const bool xm = a.vg[p].xmajor != 0;
  const int nl = xm ? a.XN : a.YN, N = xm ? a.YN : a.XN;
  const double Nd = (double)N;
  const double2* fcp = a.fc + (size_t)p * (a.U + 1);
  // x-major views integrate along x columns (line = x, k = y), the others along y rows
  const unsigned ks = (unsigned)(xm ? a.XN : 1) * (unsigned)a.ZP;  // vectors from k to k + 1
  const size_t lstride = (size_t)(xm ? 1 : a.XN) * a.ZP * VB;
  const char* img0 = reinterpret_cast<const char*>(a.img) + (size_t)(a.vb0 + ztile * ZL) * VB;  // the z-tile's first vector
  const char* img = img0 + (size_t)(active ? zi : 0) * VB;
  float* tot = s_tot + tid;
#pragma unroll
  for (int e = 0; e < CG * SV; ++e) tot[e * T::NT] = 0.f;
  Vec<SV> acc[CG];
#pragma unroll
  for (int j = 0; j < CG; ++j) vzero(acc[j]);
  int lo, hi;
  dd_warp_lines(fcp, wc0, CWW, a.U, Nd, nl, seg, nseg, lo, hi);
  const float dx = a.dx;
  // decode: lane -> channel lr (of CWW, 32 at a time) on line lc of a step of LPS
  const int LPS = CWW < 32 ? 32 / CWW : 1;
  const int lc = CWW < 32 ? lane / CWW : 0, lr0 = CWW < 32 ? lane - lc * CWW : lane;
  int rg = 0, rj = 0;
  double2 fa = make_double2(0.0, 0.0), fb = fa;
  bool uok = false;
  const auto channel = [&](int r) {
    rg = r / CG;
    rj = r - rg * CG;
    const int u = wc0 + r;
    uok = u < a.U;
    fa = __ldg(fcp + min(u, a.U));
    fb = __ldg(fcp + min(u + 1, a.U));
    fa.y += DD_MAGIC;
    fb.y += DD_MAGIC;
  };
  if (wc0 < a.U) channel(lr0);
  int since = 0;
  for (int ii0 = lo; ii0 < hi; ii0 += CC) {
    const int ncol = min(CC, hi - ii0);
    bool wide = false;
    for (int rb = 0; rb < CWW; rb += 32) {
      if (CWW > 32) channel(rb + lane);
      const bool ok = CWW > 32 ? rb + lane < CWW : lc < LPS;
#pragma unroll 1
      for (int col = lc; col < ncol && ok; col += LPS) {
        // cell and fraction of both boundaries on the line, footprint length
        const double di = (double)(ii0 + col);
        const double t0 = fma(di, fa.x, fa.y), t1 = fma(di, fb.x, fb.y);
        const DdPos p0 = dd_pos(t0, N), p1 = dd_pos(t1, N);
        const float inv = uok ? dd_rcpf((float)(t1 - t0) * dx) : 0.f;
        float w0, wm, we;
        dd_walk(p0, p1, inv, w0, wm, we);
        const int k0 = p0.k, k1 = p1.k;
        const bool up = k1 > k0;
        const int n = up ? k1 - k0 : k0 - k1;
        wide |= n > 2;
        const unsigned oe = (unsigned)k1 * ks;
        s_w[w][(col * GW + rg) * CG + rj] = make_float4(w0, wm, we, __uint_as_float(oe));
        unsigned* m = reinterpret_cast<unsigned*>(&s_m[w][col * GW + rg]);
        m[1 + rj] = n >= 2 ? DD_INNER | (unsigned)(up ? k0 + 1 : k0 - 1) * ks : 0u;
        if (rj == 0) m[0] = (unsigned)k0 * ks;
      }
    }
    wide = __any_sync(0xffffffffu, wide);
    __syncwarp();
    if (active) {
      // the start and end values of a line's walks are all loaded before the
      // first is used; a walk's interior value (one in six at the c2 geometry)
      // is loaded and added behind a branch.  Loading it ahead under a
      // predicate, or always, cost more in register moves and L1 wavefronts
      // than the wait (1.42 and 1.47 ms against 1.30 per c3 subset).
      const char* lp = img + (size_t)ii0 * lstride;
      const float4* pw = &s_w[w][g * CG];
      const uint4* pm = &s_m[w][g];
#pragma unroll 1
      for (int col = 0; col < ncol; ++col, lp += lstride, pw += GW * CG, pm += GW) {
        Vec<SV> S, E[CG];
        float4 wt[CG];
        const uint4 m = *pm;
        const unsigned om[3] = {m.y, m.z, m.w};
        vload(S, lp + (size_t)m.x * VB);
#pragma unroll
        for (int j = 0; j < CG; ++j) {
          wt[j] = pw[j];
          vload(E[j], lp + (size_t)__float_as_uint(wt[j].w) * VB);
        }
#pragma unroll
        for (int j = 0; j < CG; ++j) {
          vfma(acc[j], dup2(wt[j].x), j ? E[j - 1] : S);
          vfma(acc[j], dup2(wt[j].z), E[j]);
        }
#pragma unroll
        for (int j = 0; j < CG; ++j) {
          if ((int)om[j] < 0) {
            Vec<SV> v;
            vload(v, lp + (size_t)(om[j] & ~DD_INNER) * VB);
            vfma(acc[j], dup2(wt[j].y), v);
          }
        }
      }
      if (wide) {
        // interior values past the first (footprints over more than two cells)
        lp = img + (size_t)ii0 * lstride;
#pragma unroll 1
        for (int col = 0; col < ncol; ++col, lp += lstride) {
#pragma unroll
          for (int j = 0; j < CG; ++j) {
            const unsigned* m = reinterpret_cast<const unsigned*>(&s_m[w][col * GW + g]);
            if (!(m[1 + j] & DD_INNER)) continue;
            const float4 wt = s_w[w][(col * GW + g) * CG + j];
            const unsigned o0 = j ? __float_as_uint(s_w[w][(col * GW + g) * CG + j - 1].w) : m[0];
            const unsigned om = m[1 + j] & ~DD_INNER, oe = __float_as_uint(wt.w), st = om - o0;  // one step (mod 2^32)
            for (unsigned q = om + st; q != oe; q += st) {
              Vec<SV> v;
              vload(v, lp + (size_t)q * VB);
              vfma(acc[j], dup2(wt.y), v);
            }
          }
        }
      }
      since += ncol;
      if (since >= T::FLUSH || ii0 + CC >= hi) {
        since = 0;
#pragma unroll
        for (int j = 0; j < CG; ++j) {
#pragma unroll
          for (int s = 0; s < SV; ++s) tot[(j * SV + s) * T::NT] += vget(acc[j], s);
          vzero(acc[j]);
        }
      }
    }
    __syncwarp();
  }
  if (nseg > 1) {
    __syncthreads();
    if (seg != 0) return;
  }
  if (!active) return;
#pragma unroll
  for (int j = 0; j < CG; ++j) {
    const int u = wc0 + g * CG + j;
    if (u >= a.U) break;
    float val[SV];
#pragma unroll
    for (int s = 0; s < SV; ++s) {
      val[s] = tot[(j * SV + s) * T::NT];
      for (int q = 1; q < nseg; ++q) val[s] += tot[(j * SV + s) * T::NT + 32 * q];
    }
    dd_fwd_store<SV>(a, p, u, vb, val);
  }
}

// The same for at most 8 slices (one vector per lane and z-tile): no lanes
// share a walk, so each decodes its own two channels' walks in registers --
// three boundary cells and two footprint lengths a line -- instead of through
// shared memory.  Warp = one view x 64 channels x SV slices.
template <int SV>
__device__ __forceinline__ void fwd_thin_body(const DdFwdArgs& a, int row, int cblk, int ztile) {
  using T = DdFwdTile<SV>;
  constexpr int NW = T::NW, VB = SV * 4;
  static_assert(T::THIN_CG == 2, "the body's two channels");
  extern __shared__ float s_tot[];  // [2 * SV][NT]: this thread's totals at tid
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int nseg = a.nseg, wch = w / nseg, seg = w - wch * nseg;
  const int wc0 = (cblk * (NW / nseg) + wch) * 64;
  const int p = a.order ? a.order[row] : row;
  const int u0 = wc0 + 2 * lane, vb = a.vb0 + ztile;
  const bool xm = a.vg[p].xmajor != 0;
  const int nl = xm ? a.XN : a.YN, N = xm ? a.YN : a.XN;
  const double2* fcp = a.fc + (size_t)p * (a.U + 1);
  // neighbouring lanes read neighbouring k: x-major views from the columns
  const bool cols = xm && a.imgT;
  const size_t kstride = (size_t)(xm && !cols ? a.XN : 1) * a.ZP * VB;
  const size_t lstride = (size_t)(cols ? a.YN : (xm ? 1 : a.XN)) * a.ZP * VB;
  float* tot = s_tot + tid;
#pragma unroll
  for (int e = 0; e < 2 * SV; ++e) tot[e * T::NT] = 0.f;
  Vec<SV> acc[2];
  vzero(acc[0]);
  vzero(acc[1]);
  int lo, hi;
  dd_warp_lines(fcp, wc0, 64, a.U, (double)N, nl, seg, nseg, lo, hi);
  if (u0 < a.U) {
    const float dx = a.dx;
    double2 fl[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      fl[j] = __ldg(fcp + min(u0 + j, a.U));
      fl[j].y += DD_MAGIC;
    }
    const bool two = u0 + 1 < a.U;
    const char* lp = reinterpret_cast<const char*>(cols ? a.imgT : a.img) + (size_t)vb * VB + (size_t)lo * lstride;
    int since = 0;
#pragma unroll 2
    for (int ii = lo; ii < hi; ++ii, lp += lstride) {
      const double di = (double)ii;
      double t[3];
      DdPos pos[3];
      Vec<SV> val[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        t[j] = fma(di, fl[j].x, fl[j].y);
        pos[j] = dd_pos(t[j], N);
        vload(val[j], lp + (size_t)pos[j].k * kstride);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float inv = j == 0 || two ? dd_rcpf((float)(t[j + 1] - t[j]) * dx) : 0.f;
        float w0, wm, we;
        dd_walk(pos[j], pos[j + 1], inv, w0, wm, we);
        vfma(acc[j], dup2(w0), val[j]);
        vfma(acc[j], dup2(we), val[j + 1]);
        const int k0 = pos[j].k, k1 = pos[j + 1].k, st = k1 > k0 ? 1 : -1;
        for (int q = k0 + st; k1 != k0 && q != k1; q += st) {
          Vec<SV> v;
          vload(v, lp + (size_t)q * kstride);
          vfma(acc[j], dup2(wm), v);
        }
      }
      if (++since == T::FLUSH || ii + 1 == hi) {
        since = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
          for (int s = 0; s < SV; ++s) tot[(j * SV + s) * T::NT] += vget(acc[j], s);
          vzero(acc[j]);
        }
      }
    }
  }
  if (nseg > 1) {
    __syncthreads();
    if (seg != 0) return;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (u0 + j >= a.U) break;
    float val[SV];
#pragma unroll
    for (int s = 0; s < SV; ++s) {
      val[s] = tot[(j * SV + s) * T::NT];
      for (int q = 1; q < nseg; ++q) val[s] += tot[(j * SV + s) * T::NT + 32 * q];
    }
    dd_fwd_store<SV>(a, p, u0 + j, vb, val);
  }
}

// Allows a forward kernel its dynamic shared memory on the current device
// (above the 48 KB default with the static arrays).  Host-side, once per
// device, before any launch or capture.
template <typename K>
inline cudaError_t dd_allow_dyn(K kernel, int bytes) {
  return bytes > 0 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : cudaSuccess;
}

// One CTA per (view row, channel block, z-tile) of one call.  View rows run
// along grid x (dispatched first): the CTAs in flight are then every view of
// a few channel blocks -- rays at one distance from the centre, which miss the
// disk inside it -- instead of every channel block of a few views.  On a c3
// subset this cut the DRAM reads of the image from 2.05 to 1.33 GB per launch.
template <int SV, bool THIN>
__global__ void __launch_bounds__(256, DDFAN_DD_FWD_MIN_CTAS) k_fwd_dd(const __grid_constant__ DdFwdArgs a) {
  if constexpr (THIN) fwd_thin_body<SV>(a, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z);
  else fwd_dd_body<SV>(a, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z);
}

// One launch over a work list of many calls (batched reconstructions): CTA
// b takes item {call, view row, channel block, z-tile} = items[b].
template <int SV, bool THIN>
__global__ void __launch_bounds__(256, DDFAN_DD_FWD_MIN_CTAS) k_fwd_dd_batch(const DdFwdArgs* __restrict__ args,
                                                                             const int4* __restrict__ items) {
  const int4 it = items[blockIdx.x];
  if constexpr (THIN) fwd_thin_body<SV>(args[it.x], it.y, it.z, it.w);
  else fwd_dd_body<SV>(args[it.x], it.y, it.z, it.w);
}

// ============================================================ backprojectors

struct DdBackArgs {
  const float* q;      // residual [slot][U+1][ZP vectors of SV slices], channel U = 0
                       // (exact adjoint: weighted, r_u / |dir_u.axis|)
  int ZP;
  const ViewGeom* vg;
  int PN, U, XN, YN;
  int Z;               // slices of an output pixel
  double ocx, ocy, dx;
  // exact adjoint
  const double2* tab;  // [U] fan tangents of the boundaries (dd_edge)
  const uint16_t* lut;
  float t0, invdt, dirtf;
  int M;
  double dirt, inv_sid;
  // reference formula
  double inv_dbeta, cnt;  // cnt = detCntIdx + 1 - 0.5
  float sidf;             // source distance
  int near;               // blocks seen under a small angle: dd_block's FP32 offsets (else FP64 per voxel)
  BackEpi epi;
  int sv;              // slices per thread (the kernel's SV)
  int zl;              // lanes of a voxel group: vectors of a z-tile
  int vb0, nvb, nzt;   // first vector and vectors of [zlo, zhi); z-tiles of zl vectors
  int nseg;            // view segments a warp's views are split into (1, 2, 4 or 8)
  int thin;            // few slices: back_thin_body (zl = 1)
};

// (view, voxel block) records a warp decodes at a time (one per lane), the
// window values a record holds per pass, and a record's stride in bytes (an odd
// multiple of 16: the lanes' stores fall into different banks)
constexpr int DD_BACK_MW = 8, DD_BACK_RS = 16 * (DD_BACK_MW + 1);

template <int SV>
struct DdBackTile {
  static constexpr int NT = 256, NW = NT / 32;
  static constexpr int WBUF = 32 * DD_BACK_RS;  // bytes of window weights per warp
  static constexpr int FLUSH = 16;   // views per FP32 partial sum
  static constexpr int MIN_CTAS = SV == 4 ? DDFAN_DD_BACK_MIN_CTAS + 1 : DDFAN_DD_BACK_MIN_CTAS;
  static constexpr int STEP = 4;     // window values loaded together
  static constexpr int DYN = 4 * SV * NT * (int)sizeof(float);
};

// 2 x 2-voxel blocks: the CTA's tile is WX * GW blocks wide and WY high, its
// (8 / nseg) tile warps side by side in x while a warp's run of blocks is short
__host__ __device__ inline int dd_back_wx(int GW, int nseg) { return GW >= 8 || nseg == 8 ? 1 : 2; }

// Fractional boundary index (cell k, fraction f) of the point at v from the
// source of a view whose central ray has direction n: where it lies between
// the boundary rays along a line of the view's (constant component vl of v).
// A ray of fan tangent T has direction n + T m, m normal to n, and meets the
// line at a point that is a fractional linear function of T, so with the
// point's own tangent t and the bracket T_b <= t < T_{b+1},
//   f = 1 - (1 - (t - T_b) / (T_{b+1} - T_b)) D(T_b) / D(t),
// D(T) the line's constant component of n + T m (D(t) = vl / (n . v)) -- in exact
// arithmetic the ratio of the forward's boundary positions c_b on the line,
// from one table of all views instead of two boundary lines of this one.
// tab[b] = (T_b, 1 / (T_{b+1} - T_b)), T increasing (times dirt); lut: a guess
// of b, made exact by stepping.  nl: D(T) = nl.x + dirt T nl.y.
__device__ __forceinline__ void dd_edge(const DdBackArgs& a, const DdRay& v, bool xm, double nx, double ny, float nxf,
                                        float nyf, double nlx, double nly, int& k, float& f) {
  const double cr = nx * v.y - ny * v.x, dt = fma(nx, v.x, ny * v.y), vl = xm ? v.x : v.y;
  const float crf = nxf * v.yf - nyf * v.xf, dtf = fmaf(nxf, v.xf, nyf * v.yf), vlf = xm ? v.xf : v.yf;
  const float rf = dd_rcp_approx(dtf * vlf);
  const double r = dd_newton(dt * vl, rf), t = a.dirt * (cr * (vl * r));
  const float tf = a.dirtf * crf * (vlf * rf);
  const float m = fminf(fmaxf((tf - a.t0) * a.invdt, 0.f), (float)(a.M - 1));
  int b = min((int)__ldg(a.lut + (__float_as_int(m + 8388608.f) & 0x7fffff)), a.U - 1);
  double2 q = __ldg(a.tab + b);
  double u = (t - q.x) * q.y;
  while (u >= 1.0 && b < a.U - 1) {
    q = __ldg(a.tab + ++b);
    u = (t - q.x) * q.y;
  }
  while (u < 0.0 && b > 0) {
    q = __ldg(a.tab + --b);
    u = (t - q.x) * q.y;
  }
  k = b;
  f = __saturatef((float)fma(u - 1.0, fma(q.x, nly, nlx) * (dt * (dt * r)), 1.0));
}

// back_store for a thread's SV slices, in 16-byte pieces where the output allows.
template <int SV>
__device__ __forceinline__ void dd_back_store(const BackEpi& e, int ix, int iy, int vb, int XN, int Z, bool scale_by_mask,
                                              const float (&acc)[SV]) {
  const size_t pix = (size_t)iy * XN + ix;
  const float m = e.mask ? (float)e.mask[pix] : 1.f;
  const float cs = e.xin ? __ldg(e.colsum + pix) : 0.f;
  const size_t base = pix * Z + (size_t)vb * SV;
  const bool whole = SV >= 4 && (Z & 3) == 0 && vb * SV >= e.zlo && vb * SV + SV <= e.zhi &&
                     ((reinterpret_cast<uintptr_t>(e.out) | reinterpret_cast<uintptr_t>(e.xin)) & 15) == 0;
  float val[SV], x[SV];
#pragma unroll
  for (int s = 0; s < SV; ++s) x[s] = 0.f;
  if (e.xin) {
    if (whole) {
#pragma unroll
      for (int s = 0; s + 4 <= SV; s += 4) {
        const float4 t = *reinterpret_cast<const float4*>(e.xin + base + s);
        x[s] = t.x; x[s + 1] = t.y; x[s + 2] = t.z; x[s + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int s = 0; s < SV; ++s)
        if (vb * SV + s >= e.zlo && vb * SV + s < e.zhi) x[s] = e.xin[base + s];
    }
  }
#pragma unroll
  for (int s = 0; s < SV; ++s) {
    val[s] = scale_by_mask ? acc[s] * m : (m != 0.f ? acc[s] : 0.f);
    if (e.xin) {
      // x += t / colSum where colSum != 0, else x += t (AAPM_script/OSSART_AAPM.m:94-97)
      const float t = cs != 0.f ? __fdiv_rn(val[s], cs) : val[s];
      val[s] = x[s] + t;
      if (e.nonneg) val[s] = fmaxf(val[s], 0.f);
    }
  }
  if (whole) {
#pragma unroll
    for (int s = 0; s + 4 <= SV; s += 4)
      *reinterpret_cast<float4*>(e.out + base + s) = make_float4(val[s], val[s + 1], val[s + 2], val[s + 3]);
  } else {
#pragma unroll
    for (int s = 0; s < SV; ++s)
      if (vb * SV + s >= e.zlo && vb * SV + s < e.zhi) e.out[base + s] = val[s];
  }
}

// Positions (cell, fraction) of the two ends of voxel (px, py)'s footprint in
// view G and its weight.
template <bool ADJ>
__device__ __forceinline__ void dd_footprint(const DdBackArgs& a, const ViewGeom& G, double px, double py, float pxf,
                                             float pyf, const double2* s_at, int& kL, float& fL, int& kR, float& fR,
                                             float& wgt) {
  const double sx = G.sx, sy = G.sy;
  const float sxf = -a.sidf * G.shx, syf = -a.sidf * G.shy;
  const DdRay v{px - sx, py - sy, pxf - sxf, pyf - syf};
  if (ADJ) {
    // the voxel's two edges along the view's lines (x columns or y rows)
    const double nx = -sx * a.inv_sid, ny = -sy * a.inv_sid, hdx = 0.5 * a.dx;
    const bool xm = G.xmajor != 0;
    const double nlx = xm ? nx : ny, nly = xm ? -a.dirt * ny : a.dirt * nx;
    const double ex = xm ? 0.0 : hdx, ey = xm ? hdx : 0.0;
    const float exf = (float)ex, eyf = (float)ey;
    dd_edge(a, DdRay{v.x - ex, v.y - ey, v.xf - exf, v.yf - eyf}, xm, nx, ny, G.shx, G.shy, nlx, nly, kL, fL);
    dd_edge(a, DdRay{v.x + ex, v.y + ey, v.xf + exf, v.yf + eyf}, xm, nx, ny, G.shx, G.shy, nlx, nly, kR, fR);
    wgt = G.sgn;
  } else {
    const float l2f = fmaf(v.xf, v.xf, v.yf * v.yf);
    float l, rs;
    dd_length(l2f, l, rs);
    const bool xdom = fabs(sx) > fabs(sy);
    const double ca = fma(dd_angle(v, sx, sy, sxf, syf, s_at), a.inv_dbeta, a.cnt + DD_MAGIC);
    const double l2 = fma(v.x, v.x, v.y * v.y);
    const double da = (xdom ? v.x : v.y) * dd_newton(l2, rs * rs) * (0.5 * a.dx * a.inv_dbeta);
    wgt = (float)a.dx * l * dd_rcpf(xdom ? v.xf : v.yf);
    dd_cell(ca - da, a.U, kL, fL);
    dd_cell(ca + da, a.U, kR, fR);
  }
}

// The four footprints of a 2 x 2 block with centre (px, py).  The centre's
// position is taken in FP64; the voxels' offsets from it, a channel or two, in
// FP32 (angle between two rays from its tangent z, |z| <= 0.01: z - z^3 / 3;
// error about 1e-7 channel, against the 3e-8 the positions' fractions round
// by), which is a third of the work of four FP64 positions.  Blocks that the
// source sees under a larger angle are decoded voxel by voxel.
template <bool ADJ>
__device__ __forceinline__ void dd_block(const DdBackArgs& a, const ViewGeom& G, double px, double py, float pxf, float pyf,
                                         const double2* s_at, int (&kL)[4], float (&fL)[4], int (&kR)[4],
                                         float (&fR)[4], float (&wgt)[4]) {
  const float dxf = (float)a.dx, h = 0.5f * dxf;
  if (!a.near) {
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      int k0, k1;
      float f0, f1, w;
      const double ex = ((j & 1) - 0.5) * a.dx, ey = ((j >> 1) - 0.5) * a.dx;
      dd_footprint<ADJ>(a, G, px + ex, py + ey, pxf + (float)ex, pyf + (float)ey, s_at, k0, f0, k1, f1, w);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i == j) kL[i] = k0, fL[i] = f0, kR[i] = k1, fR[i] = f1, wgt[i] = w;
    }
    return;
  }
  const double sx = G.sx, sy = G.sy;
  const float sxf = -a.sidf * G.shx, syf = -a.sidf * G.shy;
  const DdRay v{px - sx, py - sy, pxf - sxf, pyf - syf};
  if (ADJ) {
    // six edge points: lines (columns or rows) -1/2, 1/2 and edges -1, 0, 1
    // pixels from the centre.  A point's fan tangent is the centre's plus
    // cross(v, e) / ((n . v) (n . w)), w = v + e
    const bool xm = G.xmajor != 0;
    const double nx = -sx * a.inv_sid, ny = -sy * a.inv_sid;
    const double dt = fma(nx, v.x, ny * v.y);
    const float dtf = fmaf(G.shx, v.xf, G.shy * v.yf);
    const double tc = a.dirt * (nx * v.y - ny * v.x) * dd_newton(dt, dd_rcp_approx(dtf));
    const float rdt = a.dirtf * dd_rcpf(dtf);
    const float nly = xm ? -a.dirtf * G.shy : a.dirtf * G.shx;
    int k[2][3];
    float f[2][3];
#pragma unroll
    for (int l = 0; l < 2; ++l)
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const float el = (l - 0.5f) * dxf, em = (m - 1) * dxf;
        const float ex = xm ? el : em, ey = xm ? em : el;
        const float wx = v.xf + ex, wy = v.yf + ey, dw = fmaf(G.shx, wx, G.shy * wy);
        const float dlt = (v.xf * ey - v.yf * ex) * rdt * dd_rcpf(dw);
        const double t = tc + (double)dlt;
        const float i = fminf(fmaxf(((float)t - a.t0) * a.invdt, 0.f), (float)(a.M - 1));
        int b = min((int)__ldg(a.lut + (__float_as_int(i + 8388608.f) & 0x7fffff)), a.U - 1);
        double2 q = __ldg(a.tab + b);
        float u = (float)((t - q.x) * q.y);
        while (u >= 1.f && b < a.U - 1) {
          q = __ldg(a.tab + ++b);
          u = (float)((t - q.x) * q.y);
        }
        while (u < 0.f && b > 0) {
          q = __ldg(a.tab + --b);
          u = (float)((t - q.x) * q.y);
        }
        // f = 1 - (1 - u) D(T_b) / D(t) = u + (1 - u) u (T_{b+1} - T_b) nly / D(t),
        // D(t) = vl / (n . v) of the point
        const float e = u * dd_rcp_approx((float)q.y) * nly * dw * dd_rcp_approx(xm ? wx : wy);
        k[l][m] = b;
        f[l][m] = __saturatef(fmaf(1.f - u, e, u));
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int jx = j & 1, jy = j >> 1;  // x columns: line jx, edges jy, jy + 1; y rows: line jy, edges jx, jx + 1
      kL[j] = xm ? k[jx][jy] : k[jy][jx];
      fL[j] = xm ? f[jx][jy] : f[jy][jx];
      kR[j] = xm ? k[jx][jy + 1] : k[jy][jx + 1];
      fR[j] = xm ? f[jx][jy + 1] : f[jy][jx + 1];
      wgt[j] = G.sgn;
    }
  } else {
    const bool xdom = fabs(sx) > fabs(sy);
    const double c = fma(dd_angle(v, sx, sy, sxf, syf, s_at), a.inv_dbeta, a.cnt + DD_MAGIC24);
    const int kc = max(__double2hiint(c), 0x41300000) - 0x41380000;
    const float fc = dd_fraction24(c);
    const float idb = (float)a.inv_dbeta, hdb = h * idb;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float ex = (j & 1) ? h : -h, ey = (j >> 1) ? h : -h;
      const float wx = v.xf + ex, wy = v.yf + ey;
      const float z = (v.xf * ey - v.yf * ex) * dd_rcpf(fmaf(v.xf, wx, v.yf * wy));
      const float dlt = fmaf(-z * (z * z), 1.f / 3.f, z) * idb;
      const float l2 = fmaf(wx, wx, wy * wy), ddv = xdom ? wx : wy;
      float l, rl;
      dd_length(l2, l, rl);
      const float da = ddv * (rl * rl) * hdb;
      wgt[j] = dxf * l * dd_rcpf(ddv);
      // cell and fraction of centre + offset, clamped to [0, U]
      const float r[2] = {(fc + dlt) - da, (fc + dlt) + da};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float g = (r[e] - 0.5f) + 12582912.f;  // 1.5 2^23: rounds to the cell (a fraction of 1 may stay below)
        int k = kc + (__float_as_int(g) - 0x4b400000);
        float f = r[e] - (g - 12582912.f);
        if ((unsigned)k >= (unsigned)a.U) {
          f = k < 0 ? 0.f : 1.f;
          k = k < 0 ? 0 : a.U - 1;
        }
        if (e) kR[j] = k, fR[j] = f;
        else kL[j] = k, fL[j] = f;
      }
    }
  }
}

// A thread's totals (4 voxels x SV slices), cleared; whether any is infinite or
// NaN.  Where one is, the views are summed again value by value ("careful"): a
// window value outside a voxel's footprint has weight 0 for that voxel, and 0
// times an infinite or NaN value is NaN.  So such a value reaches the voxels
// whose footprints hold it and no others, and finite data are summed once.  The
// wide kernel takes its loop again, with the decode's one copy of the code: a
// function of its own, called at the end, cost the REF kernel 5 % (0.93 -> 0.98
// ms per c3 subset).  The thin one has the loop twice: the branch in it cost 2 %
// (one slice of 256^2, 123 views, exact adjoint: 113 -> 115 us).
template <int SV>
__device__ __forceinline__ void back_dd_clear(float* tot) {
#pragma unroll
  for (int e = 0; e < 4 * SV; ++e) tot[e * DdBackTile<SV>::NT] = 0.f;
}
template <int SV>
__device__ __forceinline__ bool back_dd_nonfinite(const float* tot) {
  bool bad = false;
#pragma unroll
  for (int e = 0; e < 4 * SV; ++e) bad = bad || !(fabsf(tot[e * DdBackTile<SV>::NT]) <= 3.402823466e38f);
  return bad;
}

// Measured per c3 subset (96 views x 736 channels, 512^2 x 128): reference
// formula 1.40 -> 0.91 ms, exact adjoint 1.77 -> 1.05 ms (0.86 ms of either
// when the decode is left out); 1111 views of 384^2 x 45, exact adjoint 10.8 ->
// 5.0 ms.  With each voxel decoded by itself (1.08 and 1.25 ms), 16 warps an SM at 128 registers with 4 values in flight each beat 24
// at 80 with 1 (1.20), 3 (1.29) or 4 (1.14): more warps spread over more views
// and lose the L1 hits (80 -> 68 %).
//
// Both backprojectors.  A voxel's sample of a view is Phi(cR) - Phi(cL), Phi
// the channel prefix sum of the residual: of its two pixel edges along the
// view's lines for the exact adjoint (the transpose of k_fwd_dd: pixel k of
// line ii receives sum_u w_u (fraction of footprint u inside [k, k+1]) =
// Q(beta(k+1)) - Q(beta(k)), beta the fractional boundary index of an edge),
// of its angular footprint for the reference's formula (MultiSlicesBackGPU.cu:
// 115-184: alpha -+ da, da = dx ddv / (2 l^2), weight dx l / ddv).
//
// What bounds it is the L1 pipe and instruction issue, not DRAM: a voxel and
// view need two or three residual values of 128 slices, and neighbouring
// voxels mostly the same ones.  So a thread owns a 2 x 2 block of voxels x SV
// slices and, per view, reads the window of channels the block's four
// footprints cover once (3.2 values at the c2 geometry where four voxels on
// their own read 8.8), each value weighted into all four sums: the decode
// writes the four overlap weights of every window value to shared memory, so
// the inner loop is one value load, one weight load and 4 SV FMAs, with no
// address or branch per voxel.  It needs no view order and takes both view
// orientations in one pass.  Windows of any width work: a record holds 8
// values at a time, wider ones take more passes.  Sums are kept per FLUSH
// views and added to totals in shared memory, so a sum over thousands of
// views rounds like one over a few; with nseg > 1 the views are split over
// warps whose totals are added at the end.
template <int SV, bool ADJ>
__device__ __forceinline__ void back_dd_body(const DdBackArgs& a, int tile, int ztile) {
  using T = DdBackTile<SV>;
  constexpr int NW = T::NW, VB = SV * 4;
  __shared__ __align__(16) unsigned char s_wt[NW][T::WBUF];
  __shared__ uint2 s_h[NW][32];  // record: window start (vectors), values in this pass
  __shared__ double2 s_at[ADJ ? 1 : 2 * DD_ATAN_N + 1];
  extern __shared__ float s_tot[];  // [4 * SV][NT]: this thread's totals at tid
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int ZL = a.zl, GW = 32 / ZL;
  const int g = lane / ZL, zi = lane - g * ZL;
  const int nseg = a.nseg, wt = w / nseg, seg = w - wt * nseg;
  const int WX = dd_back_wx(GW, nseg), WY = (NW / nseg) / WX;
  const int ntx = ((a.XN + 1) / 2 + WX * GW - 1) / (WX * GW);
  const int ty = tile / ntx, tx = tile - ty * ntx;
  const int bx0 = (tx * WX + wt % WX) * GW, y0 = 2 * (ty * WY + wt / WX);  // the warp's first block; its rows y0, y0 + 1
  const int vb = a.vb0 + ztile * ZL + zi;
  const int x0 = 2 * (bx0 + g);
  const bool active = g < GW && ztile * ZL + zi < a.nvb && x0 < a.XN && y0 < a.YN;
  constexpr int MW = DD_BACK_MW, RS = DD_BACK_RS;
  const int VC = 32 / GW;  // views decoded at a time
  const size_t vstride = (size_t)(a.U + 1) * a.ZP * VB, kstride = (size_t)a.ZP * VB;
  const char* q = reinterpret_cast<const char*>(a.q) + (size_t)(active ? vb : 0) * VB;
  if (!ADJ) {
    for (int j = tid; j <= 2 * DD_ATAN_N; j += T::NT) s_at[j] = dd_atan_entry(j);
    __syncthreads();
  }
  float* tot = s_tot + tid;
  Vec<SV> acc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) vzero(acc[j]);
  // decode: lane -> block lb of view lv of VC
  const int lv = lane / GW, lb = lane - lv * GW;
  const double px = (2 * (bx0 + lb) + 0.5 - a.ocx) * a.dx, py = (y0 + 0.5 - a.ocy) * a.dx;
  const float pxf = (float)px, pyf = (float)py;
  bool on[4], von = false;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int xx = 2 * (bx0 + lb) + (j & 1), yy = y0 + (j >> 1);
    on[j] = lv < VC && xx < a.XN && yy < a.YN && (!a.epi.mask || a.epi.mask[(size_t)yy * a.XN + xx] != 0);
    von = von || on[j];
  }
  const int vbeg = (int)((long long)a.PN * seg / nseg), vend = (int)((long long)a.PN * (seg + 1) / nseg);
  for (bool careful = false;; careful = true) {
    back_dd_clear<SV>(tot);
    int since = 0;
    for (int v0 = vbeg; v0 < vend; v0 += VC) {
      const int nvc = min(VC, vend - v0);
      int mmax = 0;
      for (int i0 = 0; i0 == 0 || i0 < mmax; i0 += MW) {  // windows wider than a record: more passes
        if (lv < nvc) {
          int kL[4], kR[4], m = 0, kb = 0x7fffffff, ke = -1;
          float fL[4], fR[4], wgt[4];
          if (von) {
            dd_block<ADJ>(a, a.vg[v0 + lv], px, py, pxf, pyf, s_at, kL, fL, kR, fR, wgt);
            // the block's window: the cells its footprints cover
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (on[j]) {
                kb = min(kb, min(kL[j], kR[j]));
                ke = max(ke, max(kL[j], kR[j]));
              } else {
                wgt[j] = 0.f;
              }
            }
            // whole steps: more values, with weight 0, after the window or, at the
            // detector's end, before it
            m = (ke - kb + T::STEP) / T::STEP * T::STEP;
            kb = max(min(kb, a.U + 1 - m), 0);
          } else {
            kb = 0;
          }
          mmax = max(mmax, m);
          const int n = min(max(m - i0, 0), MW);
          if (n) {
            // the value in cell k has the weight of [cL, cR]'s part inside
            // [k, k + 1] (negative where cR < cL): sat(cR - k) - sat(cL - k), the
            // cells' difference exact
            float dL[4], dR[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              dL[j] = (float)(kL[j] - kb - i0);
              dR[j] = (float)(kR[j] - kb - i0);
            }
            float4* wp = reinterpret_cast<float4*>(&s_wt[w][lane * RS]);
#pragma unroll 1
            for (int i = 0; i < n; ++i, ++wp) {
              float x[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                x[j] = (__saturatef(dR[j] + fR[j]) - __saturatef(dL[j] + fL[j])) * wgt[j];
                dL[j] -= 1.f;
                dR[j] -= 1.f;
              }
              *wp = make_float4(x[0], x[1], x[2], x[3]);
            }
          }
          s_h[w][lane] = make_uint2((unsigned)(lv * (a.U + 1) + kb + (n ? i0 : 0)) * (unsigned)a.ZP, (unsigned)n);
        }
        mmax = __reduce_max_sync(0xffffffffu, mmax);
        __syncwarp();
        if (active) {
          const char* qc = q + (size_t)v0 * vstride;
          const uint2* hp = &s_h[w][g];
          const unsigned char* rp = &s_wt[w][g * RS];
#pragma unroll 1
          for (int vv = 0; vv < nvc; ++vv, hp += GW, rp += GW * RS) {
            const uint2 h = *hp;
            const float4* wp = reinterpret_cast<const float4*>(rp);
            const char* qp = qc + (size_t)h.x * VB;
            if (careful) {
#pragma unroll 1
              for (int i = (int)h.y; i > 0; --i, qp += kstride, ++wp) {
                Vec<SV> val;
                vload(val, qp);
                if (wp->x != 0.f) vfma(acc[0], dup2(wp->x), val);
                if (wp->y != 0.f) vfma(acc[1], dup2(wp->y), val);
                if (wp->z != 0.f) vfma(acc[2], dup2(wp->z), val);
                if (wp->w != 0.f) vfma(acc[3], dup2(wp->w), val);
              }
              continue;
            }
#pragma unroll 1
            for (int i = (int)h.y; i > 0; i -= T::STEP, qp += T::STEP * kstride, wp += T::STEP) {
              Vec<SV> val[T::STEP];
#pragma unroll
              for (int t = 0; t < T::STEP; ++t) vload(val[t], qp + t * kstride);
#pragma unroll
              for (int t = 0; t < T::STEP; ++t) {
                const float4 ww = wp[t];
                vfma(acc[0], dup2(ww.x), val[t]);
                vfma(acc[1], dup2(ww.y), val[t]);
                vfma(acc[2], dup2(ww.z), val[t]);
                vfma(acc[3], dup2(ww.w), val[t]);
              }
            }
          }
        }
        __syncwarp();
      }
      since += nvc;
      if (since >= T::FLUSH || v0 + VC >= vend) {
        since = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int s = 0; s < SV; ++s) tot[(j * SV + s) * T::NT] += vget(acc[j], s);
          vzero(acc[j]);
        }
      }
    }
    if (careful || !__any_sync(0xffffffffu, back_dd_nonfinite<SV>(tot))) break;
  }
  if (nseg > 1) {
    __syncthreads();
    if (seg != 0) return;
  }
  if (!active) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int ix = x0 + (j & 1), iy = y0 + (j >> 1);
    if (ix >= a.XN || iy >= a.YN) continue;
    float val[SV];
#pragma unroll
    for (int s = 0; s < SV; ++s) {
      val[s] = tot[(j * SV + s) * T::NT];
      for (int r = 1; r < nseg; ++r) val[s] += tot[(j * SV + s) * T::NT + 32 * r];
    }
    dd_back_store<SV>(a.epi, ix, iy, vb, a.XN, a.Z, ADJ, val);
  }
}

// The same for at most 8 slices (one vector per lane and z-tile): no lanes
// share a block, so each decodes its own in registers and weights the window
// values as it loads them.
template <int SV, bool ADJ>
__device__ __forceinline__ void back_thin_body(const DdBackArgs& a, int tile, int ztile) {
  using T = DdBackTile<SV>;
  constexpr int NW = T::NW, VB = SV * 4;
  __shared__ double2 s_at[ADJ ? 1 : 2 * DD_ATAN_N + 1];
  extern __shared__ float s_tot[];  // [4 * SV][NT]: this thread's totals at tid
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int nseg = a.nseg, wt = w / nseg, seg = w - wt * nseg;
  const int nbx = (a.XN + 1) / 2, nby = (a.YN + 1) / 2;
  const int bi = (tile * (NW / nseg) + wt) * 32 + lane;  // the lane's block
  const int by = bi / nbx, bx = bi - by * nbx;
  const int vb = a.vb0 + ztile;
  if (!ADJ) {
    for (int j = tid; j <= 2 * DD_ATAN_N; j += T::NT) s_at[j] = dd_atan_entry(j);
    __syncthreads();
  }
  float* tot = s_tot + tid;
  Vec<SV> acc[4];
  bool on[4], any = false;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    vzero(acc[j]);
    const int ix = 2 * bx + (j & 1), iy = 2 * by + (j >> 1);
    on[j] = by < nby && ix < a.XN && iy < a.YN && (!a.epi.mask || a.epi.mask[(size_t)iy * a.XN + ix] != 0);
    any = any || on[j];
  }
  const double px = (2 * bx + 0.5 - a.ocx) * a.dx, py = (2 * by + 0.5 - a.ocy) * a.dx;
  const float pxf = (float)px, pyf = (float)py;
  const int vbeg = (int)((long long)a.PN * seg / nseg), vend = (int)((long long)a.PN * (seg + 1) / nseg);
  const size_t kstride = (size_t)a.ZP * VB, vstride = (size_t)(a.U + 1) * kstride;
  const char* q0 = reinterpret_cast<const char*>(a.q) + (size_t)vb * VB + (size_t)vbeg * vstride;
  const auto views = [&](auto careful) {
    back_dd_clear<SV>(tot);
    const char* q = q0;
    int since = 0;
    for (int p = vbeg; any && p < vend; ++p, q += vstride) {
      float fL[4], fR[4], wgt[4];
      int kL[4], kR[4], kb = 0x7fffffff, ke = -1;
      dd_block<ADJ>(a, a.vg[p], px, py, pxf, pyf, s_at, kL, fL, kR, fR, wgt);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (on[j]) {
          kb = min(kb, min(kL[j], kR[j]));
          ke = max(ke, max(kL[j], kR[j]));
        } else {
          wgt[j] = 0.f;
        }
      }
      // the value in cell k has the weight of [cL, cR]'s part inside [k, k + 1]:
      // sat(cR - k) - sat(cL - k), the cells' difference exact
      float dL[4], dR[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dL[j] = (float)(kL[j] - kb);
        dR[j] = (float)(kR[j] - kb);
      }
      const char* qp = q + (size_t)kb * kstride;
#pragma unroll 2
      for (int k = kb; k <= ke; ++k, qp += kstride) {
        Vec<SV> v;
        vload(v, qp);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float x = (__saturatef(dR[j] + fR[j]) - __saturatef(dL[j] + fL[j])) * wgt[j];
          if (!decltype(careful)::value || x != 0.f) vfma(acc[j], dup2(x), v);
          dL[j] -= 1.f;
          dR[j] -= 1.f;
        }
      }
      if (++since == T::FLUSH || p + 1 == vend) {
        since = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int s = 0; s < SV; ++s) tot[(j * SV + s) * T::NT] += vget(acc[j], s);
          vzero(acc[j]);
        }
      }
    }
  };
  views(std::false_type());
  if (back_dd_nonfinite<SV>(tot)) views(std::true_type());
  if (nseg > 1) {
    __syncthreads();
    if (seg != 0) return;
  }
  if (by >= nby) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int ix = 2 * bx + (j & 1), iy = 2 * by + (j >> 1);
    if (ix >= a.XN || iy >= a.YN) continue;
    float val[SV];
#pragma unroll
    for (int s = 0; s < SV; ++s) {
      val[s] = tot[(j * SV + s) * T::NT];
      for (int r = 1; r < nseg; ++r) val[s] += tot[(j * SV + s) * T::NT + 32 * r];
    }
    dd_back_store<SV>(a.epi, ix, iy, vb, a.XN, a.Z, ADJ, val);
  }
}

// One CTA per (voxel tile, z-tile) of one call.
template <int SV, bool ADJ, bool THIN>
__global__ void __launch_bounds__(256, DdBackTile<SV>::MIN_CTAS) k_back_dd(const __grid_constant__ DdBackArgs a) {
  if constexpr (THIN) back_thin_body<SV, ADJ>(a, (int)blockIdx.x, (int)blockIdx.z);
  else back_dd_body<SV, ADJ>(a, (int)blockIdx.x, (int)blockIdx.z);
}

// The work-list launch: CTA b takes item {call, voxel tile, z-tile} = items[b].
// The call's arguments are read from shared memory, where the grid kernel has
// them in the constant bank: read in place from global memory they stayed in
// registers (16 solves of 256^2 x 16, 720 views, an iteration of all: 37.5 ->
// 34.8 ms; 32 of 256^2 x 8, 360 views: 24.7 -> 23.2).
template <int SV, bool ADJ, bool THIN>
__global__ void __launch_bounds__(256, DdBackTile<SV>::MIN_CTAS) k_back_dd_batch(const DdBackArgs* __restrict__ args,
                                                                                 const int4* __restrict__ items) {
  __shared__ __align__(16) unsigned s_args[sizeof(DdBackArgs) / 4];
  static_assert(sizeof(DdBackArgs) % 4 == 0 && alignof(DdBackArgs) <= 16, "copied by words");
  const int4 it = items[blockIdx.x];
  const unsigned* src = reinterpret_cast<const unsigned*>(args + it.x);
  for (int i = threadIdx.x; i < (int)(sizeof(DdBackArgs) / 4); i += 256) s_args[i] = src[i];
  __syncthreads();
  const DdBackArgs& a = *reinterpret_cast<const DdBackArgs*>(s_args);
  if constexpr (THIN) back_thin_body<SV, ADJ>(a, it.y, it.z);
  else back_dd_body<SV, ADJ>(a, it.y, it.z);
}

// ============================================================ dispatch

// go(SV, THIN) with the constants of a call: 8 or 4 slices per thread, and for
// few slices the thin kernels (1 slice: thin only)
template <class F>
inline void dd_dispatch(int sv, int thin, F&& go) {
  using I8 = std::integral_constant<int, 8>;
  using I4 = std::integral_constant<int, 4>;
  using I1 = std::integral_constant<int, 1>;
  if (sv == 1) go(I1(), std::true_type());
  else if (sv == 4) thin ? go(I4(), std::true_type()) : go(I4(), std::false_type());
  else thin ? go(I8(), std::true_type()) : go(I8(), std::false_type());
}

// ============================================================ staging

// dst[pix][z] = z < Z ? src[pix][z] * mask[pix] : 0 for za <= z < zb of Zp
// slices (mask, src null = 1): the masked image with its slices padded, or the
// vectors of a slice range of it.
static __global__ void k_stage_image(const float* __restrict__ src, int Z, const uint8_t* __restrict__ mask,
                                     float* __restrict__ dst, int Zp, size_t npix, int za, int zb) {
  const int nz = zb - za;
  const size_t n = npix * nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t pix = i / nz;
    const int z = za + (int)(i - pix * nz);
    float v = 0.f;
    if (z < Z) {
      v = src ? src[pix * Z + z] : 1.f;
      if (mask && mask[pix] == 0) v = 0.f;
    }
    dst[pix * Zp + z] = v;
  }
}

// out[x][y][z] = in[y][x][z] for pixels of P float4: 32 x 32 pixels a CTA
static __global__ void __launch_bounds__(256) k_columns(const float4* __restrict__ in, float4* __restrict__ out, int XN,
                                                        int YN, int P) {
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  for (int e = threadIdx.x; e < 32 * 32 * P; e += 256) {
    const int z = e % P, i = e / P, y = y0 + (i & 31), x = x0 + (i >> 5);
    if (x < XN && y < YN) out[((size_t)x * YN + y) * P + z] = __ldg(in + ((size_t)y * XN + x) * P + z);
  }
}

// The same for many images in one launch (batched reconstructions): CTA b takes
// item {image, 32-pixel column block, row block} = items[b].
struct ColArgs {
  const float* in;
  float* out;
  int XN, YN, Zs;  // Zs = 1, or a multiple of 4
};
static __global__ void __launch_bounds__(256) k_columns_batch(const ColArgs* __restrict__ args, const int4* __restrict__ items) {
  __shared__ float t[32][33];
  const int4 it = items[blockIdx.x];
  const ColArgs a = args[it.x];
  const int x0 = it.y * 32, y0 = it.z * 32;
  if (a.Zs == 1) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = w; i < 32; i += 8)
      if (y0 + i < a.YN && x0 + lane < a.XN) t[i][lane] = a.in[(size_t)(y0 + i) * a.XN + x0 + lane];
    __syncthreads();
    for (int i = w; i < 32; i += 8)
      if (x0 + i < a.XN && y0 + lane < a.YN) a.out[(size_t)(x0 + i) * a.YN + y0 + lane] = t[lane][i];
    return;
  }
  const int P = a.Zs / 4;
  const float4* in = reinterpret_cast<const float4*>(a.in);
  float4* out = reinterpret_cast<float4*>(a.out);
  for (int e = threadIdx.x; e < 32 * 32 * P; e += 256) {
    const int z = e % P, i = e / P, y = y0 + (i & 31), x = x0 + (i >> 5);
    if (x < a.XN && y < a.YN) out[((size_t)x * a.YN + y) * P + z] = in[((size_t)y * a.XN + x) * P + z];
  }
}

// dst[p][u][z] = src[p][u][z] * wgt[p][u] for u < U, z < Z; zero on the
// guard channel u = U, on padding slices and on DD_PAST entries past the last
// view (wgt, src null = 1); za <= z < zb of Zp slices.
static __global__ void k_stage_sino(const float* __restrict__ src, int Z, const float* __restrict__ wgt, int U,
                                    float* __restrict__ dst, int Zp, size_t PN, int za, int zb) {
  const int nz = zb - za;
  const size_t n = (PN * (U + 1) + DD_PAST) * nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / nz;
    const int z = za + (int)(i - r * nz);
    const size_t p = r / (U + 1);
    const int u = (int)(r - p * (U + 1));
    float v = 0.f;
    if (u < U && z < Z && p < PN) {
      const size_t e = p * U + u;
      v = src ? src[e * Z + z] : 1.f;
      if (wgt) v *= wgt[e];
    }
    dst[r * Zp + z] = v;
  }
}

// The published image of a solver that keeps masked voxels at 0 internally:
// out[pix][z] = mask ? x[pix][z] : x0[pix][z], clamped at 0 when the updates
// clamp (every update leaves a masked voxel at its initial value).
static __global__ void k_publish_masked(const float* __restrict__ x, int Zi, const float* __restrict__ x0,
                                        int Z, const uint8_t* __restrict__ mask, int clamp0,
                                        float* __restrict__ out, size_t npix) {
  const size_t n = npix * Z;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t pix = i / Z;
    const int z = (int)(i - pix * Z);
    float v;
    if (!mask || mask[pix] != 0) {
      v = x[pix * Zi + z];
    } else {
      v = x0[i];
      if (clamp0) v = fmaxf(v, 0.f);
    }
    out[i] = v;
  }
}

}  // namespace ddfan
