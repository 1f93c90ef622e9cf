// gpv_rows.cuh -- rows of cells that a triangle's SAT passes, solved instead of tested: the range
// arithmetic shared by the Level1 kernel, the Level2 SAT and fill, and the Level2 normals.  Nothing here
// decides a state by itself: every bound is wider than the float tests' own error, and what lies between
// the inner and the outer bound runs the exact predicates of gpv_common.cuh.
#pragma once
#include "gpv_common.cuh"

namespace gpv {

constexpr float EPS24 = 5.9604644775390625e-08f;  // 2^-24

// 1/x to about an ulp (range arithmetic only, never inside a predicate).
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ff(float a, float b, float c) { return __fmaf_rn(a, b, c); }

__device__ __forceinline__ uint32_t cvt_pair_ceil(float lo, float hi) {
  short a, b;  // (the conversion saturates)
  asm("cvt.rpi.s16.f32 %0, %1;" : "=h"(a) : "f"(lo));
  asm("cvt.rpi.s16.f32 %0, %1;" : "=h"(b) : "f"(hi));
  return (uint32_t)(uint16_t)a | ((uint32_t)(uint16_t)b << 16);
}
__device__ __forceinline__ uint32_t cvt_pair_floor(float lo, float hi) {
  short a, b;
  asm("cvt.rmi.s16.f32 %0, %1;" : "=h"(a) : "f"(lo));
  asm("cvt.rmi.s16.f32 %0, %1;" : "=h"(b) : "f"(hi));
  return (uint32_t)(uint16_t)a | ((uint32_t)(uint16_t)b << 16);
}

// ---- rows of a two-dimensional triangle / square test ----------------------------------------
// The squares of half sizes (ha, hb) centred at ((i - base) ga, k gb); the triangle (a[], b[]).
// An edge (ea, eb) separates where eb * a - ea * b of the edge (t, at the square) and of the opposite
// vertex (t + S) both exceed rad = |eb| ha + |ea| hb or both lie below -rad, so it passes for
//   t0 + k ea gb - rad + min(S, 0)  <=  (i - base) eb ga  <=  t0 + k ea gb + rad + max(S, 0),
// t0 being t at (0, 0).  `dl` bounds the roundings of those sides and of what the float test compares
// (see the callers), ta and tb the distance of the centre tables from their affine form; a slope below
// 1/512 of the bound is replaced by it, which moves a side by at most 1/16 of it over 32 cells.  kIdx
// covers the rounding of the index arithmetic (values up to 64 with a relative error of a few 2^-23).
// Row k passes the edge's float test for every i in [lo + w2, hi - w2] and for none outside [lo, hi],
// with lo and hi moving by s per row.
constexpr float kIdx = 1.f / 16384.f;
struct EdgeRows { float lo, hi, w2, s; };

__device__ __forceinline__ EdgeRows edge_rows(float ea, float eb, float a, float b, float ha, float hb,
                                              float ga, float gb, float sn, float sp, float dl,
                                              float ta, float tb, float base) {
  const float t = ff(eb, a, -(ea * b));
  const float rad = ff(fabsf(eb), ha, fabsf(ea) * hb);
  const float d = ff(fabsf(eb), ta, ff(fabsf(ea), tb, dl));
  const float s = eb * ga;
  const float inv = rcp_fast(copysignf(fmaxf(fabsf(s), d * (1.f / 512.f)), s));
  const float x1 = (t - rad + sn) * inv, x2 = (t + rad + sp) * inv;
  const float w = ff(d, fabsf(inv), kIdx);
  return {fminf(x1, x2) - w + base, fmaxf(x1, x2) + w + base, 2.f * w, ea * gb * inv};
}

// Solves rows 0 .. n-1 into out[] and returns the number of cells that can pass.  A row's [lo_o, end_o)
// holds every i that can pass, [lo_i, end_i) only ones that do; one byte each, lo_o | lo_i << 8 | end_i << 16 | end_o << 24.  bl and be are the
// i that can and that certainly pass the a axis' own test (lo_o | lo_i << 16 and end_i | end_o << 16),
// and rows outside [in_lo, in_end) may fail the b axis' own: they pass nothing for certain.
__device__ __forceinline__ uint32_t solve_rows(uint32_t *out, int n, float a0, float a1, float a2, float b0,
                                           float b1, float b2, float ha, float hb, float ga, float gb,
                                           float dl, float ta, float tb, int base, uint32_t bl,
                                           uint32_t be, int in_lo, int in_end) {
  const float e0a = a1 - a0, e0b = b1 - b0, e1a = a2 - a1, e1b = b2 - b1, e2a = a0 - a2, e2b = b0 - b2;
  const float S = ff(e0b, e1a, -(e0a * e1b));
  const float sn = fminf(S, 0.f), sp = fmaxf(S, 0.f), fb = (float)base;
  const EdgeRows r0 = edge_rows(e0a, e0b, a0, b0, ha, hb, ga, gb, sn, sp, dl, ta, tb, fb);
  const EdgeRows r1 = edge_rows(e1a, e1b, a1, b1, ha, hb, ga, gb, sn, sp, dl, ta, tb, fb);
  const EdgeRows r2 = edge_rows(e2a, e2b, a2, b2, ha, hb, ga, gb, sn, sp, dl, ta, tb, fb);
  float k = 0.f;
  uint32_t cells = 0;
#pragma unroll 1
  for (int i = 0; i < n; ++i, k += 1.f) {
    const float l0 = ff(k, r0.s, r0.lo), l1 = ff(k, r1.s, r1.lo), l2 = ff(k, r2.s, r2.lo);
    const float h0 = ff(k, r0.s, r0.hi), h1 = ff(k, r1.s, r1.hi), h2 = ff(k, r2.s, r2.hi);
    const float lo_o = fmaxf(l0, fmaxf(l1, l2)), hi_o = fminf(h0, fminf(h1, h2));
    const float lo_i = fmaxf(l0 + r0.w2, fmaxf(l1 + r1.w2, l2 + r2.w2));
    const float hi_i = fminf(h0 - r0.w2, fminf(h1 - r1.w2, h2 - r2.w2));
    const uint32_t L = __vmins2(__vmaxs2(cvt_pair_ceil(lo_o, lo_i), bl), 0x00400040u);
    uint32_t E = __vmaxs2(__vmins2(cvt_pair_floor(hi_i + 1.f, hi_o + 1.f), be), 0u);
    if (i < in_lo || i >= in_end) E &= 0xffff0000u;
    out[i] = __byte_perm(L, E, 0x6420);
    cells += (uint32_t)max((int)E >> 16, (int)(L & 0xffffu)) - (L & 0xffffu);
  }
  return cells;
}

// Lists a triangle's sub-columns (slot | row << 5 | column << 10, both from the triangle's first, | certain
// to pass the x/y tests << 15) in rows [d0, d1) from its solved x/y rows (nullptr: all np x nq, none certain).
__device__ __forceinline__ void list_columns(uint16_t *out, const uint32_t *xy, int slot, int p0, int np,
                                             int d0, int d1) {
#pragma unroll 1
  for (int dq = d0; dq < d1; ++dq) {
    const uint32_t w = xy ? xy[dq] : (uint32_t)(p0 | ((p0 + np) << 24));
    const int lo_i = (int)((w >> 8) & 255u), end_i = (int)((w >> 16) & 255u), end = (int)(w >> 24);
    const uint32_t e = (uint32_t)(slot | (dq << 5));
#pragma unroll 1
    for (int p = (int)(w & 255u); p < end; ++p)
      *out++ = (uint16_t)(e | (uint32_t)((p - p0) << 10) | (p >= lo_i && p < end_i ? 0x8000u : 0u));
  }
}

// Cells of one axis whose boxes can meet [tmin, tmax] ([lo, hi]) and those that certainly do
// ([in_lo, in_end)), by the SAT's own box-axis test; `md` (cells) bounds the distance of the centre
// table from c0 + k * g2 and the roundings.  Where inv_g2 overflows (cells under 2^-128) the values are
// infinite or not numbers: every cell can then meet the box and none does for certain.
__device__ __forceinline__ void cell_ranges(float tmin, float tmax, float c0, float inv_g2, int n2,
                                            float md, int &lo, int &hi, int &in_lo, int &in_end) {
  const float f0 = ff(tmin - c0, inv_g2, 0.5f), f1 = ff(tmax - c0, inv_g2, 0.5f);
  const float last = (float)(n2 - 1);
  lo = max(__float2int_rd(f0 - md), 0);
  hi = __float2int_rd(fminf(f1 + md, last));
  in_lo = __float2int_rd(fmaxf(fminf(f0 + md, last + 1.f), 0.f));
  in_end = __float2int_rd(fminf(fmaxf(f1 - md, -1.f), last)) + 1;
}

}  // namespace gpv
