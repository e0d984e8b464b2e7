// Ray coordinates from (hi, lo) float coefficients. Device code only.
#pragma once
#include "kernels.h"

namespace risa_gb {

// Window of an angle for a tile whose lowest coordinate is at pixel (cx, cy):
// its first bin w0 (a multiple of ALIGN) and the lowest coordinate relative to
// it, t0 + cx a + cy b - w0 >= 0. Error-free FP32 sums (Knuth's two-sum) and
// products of the (hi, lo) coefficients keep ~2^-40 of a bin; FP64 has few units
// per SM (one slice of 1024 x 1024 -> 512^2: 148 us with FP64 windows, 142 with
// these). The sum u + lo, rounded, may reach an integer that the coordinate lies
// just below (by up to half a unit of u, 3e-5 of a bin at 1000 bins): the floor is
// then one less. So the window is FP64's and rel is as near as FP64 rounded to FP32.
template <int ALIGN>
__device__ __forceinline__ void patch_window(const BPPatchAngle& t, int cx, int cy, int* w0, float* rel) {
   const float x = (float)cx, y = (float)cy;
   const float p = __fmul_rn(x, t.a_hi), q = __fmul_rn(y, t.b_hi);
   const float pe = fmaf(x, t.a_lo, fmaf(x, t.a_hi, -p)), qe = fmaf(y, t.b_lo, fmaf(y, t.b_hi, -q));
   const float s = __fadd_rn(t.t0_hi, p), sv = __fsub_rn(s, t.t0_hi);
   const float se = __fadd_rn(__fsub_rn(t.t0_hi, __fsub_rn(s, sv)), __fsub_rn(p, sv));
   const float u = __fadd_rn(s, q), uv = __fsub_rn(u, s);
   const float ue = __fadd_rn(__fsub_rn(s, __fsub_rn(u, uv)), __fsub_rn(q, uv));
   const float lo = __fadd_rn(__fadd_rn(se, ue), __fadd_rn(__fadd_rn(pe, qe), t.t0_lo));
   float w = floorf(__fadd_rn(u, lo));
   if (__fadd_rn(__fsub_rn(u, w), lo) < 0.f) w -= 1.f;
   *w0 = (int)w & ~(ALIGN - 1);
   *rel = __fadd_rn(__fsub_rn(u, (float)*w0), lo);
}

}  // namespace risa_gb
