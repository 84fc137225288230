// Order-5 B-splines of the PME sites: the table of every slot's grid origin,
// spline values and derivatives, formed once per position update
// (k_scatter_pos) and read by the spread and gather kernels (pme.cu).
// Weights as bsplgen (include/seq/bsplgen.h:27-116), grid origins as
// src/cu/pme.cu:31-58.
#pragma once
#include "common.cuh"

namespace t9gb {

// Piece j of the cardinal B-spline M5 and its first three derivatives at
// the site's fraction w, as polynomials.  M5 is even about its centre: the
// first two pieces are the last two at t = 1 - w with the odd derivatives'
// sign flipped, so there is no cancellation at either end.  Coefficients
// x 24: centre 11 + 12 t - 6 t^2 - 12 t^3 + 6 t^4, next 1 + 4 t + 6 t^2 +
// 4 t^3 - 4 t^4, edge t^4.
template <int J>
__device__ __forceinline__ void spline_piece(float w, float* th)
{
   constexpr bool mid = J == 2, edge = J == 0 || J == 4, mirror = J < 2;
   constexpr float q = 1.f / 24.f;
   constexpr float c0 = mid ? 11.f * q : edge ? 0.f : q;
   constexpr float c1 = mid ? 12.f * q : edge ? 0.f : 4.f * q;
   constexpr float c2 = mid ? -6.f * q : edge ? 0.f : 6.f * q;
   constexpr float c3 = mid ? -12.f * q : edge ? 0.f : 4.f * q;
   constexpr float c4 = mid ? 6.f * q : edge ? q : -4.f * q;
   const float t = mirror ? 1.f - w : w;
   th[0] = __fmaf_rn(__fmaf_rn(__fmaf_rn(__fmaf_rn(c4, t, c3), t, c2), t, c1), t, c0);
   const float d1 = __fmaf_rn(__fmaf_rn(__fmaf_rn(4.f * c4, t, 3.f * c3), t, 2.f * c2), t, c1);
   th[1] = mirror ? -d1 : d1;
   th[2] = __fmaf_rn(__fmaf_rn(12.f * c4, t, 6.f * c3), t, 2.f * c2);
   const float d3 = __fmaf_rn(24.f * c4, t, 6.f * c3);
   th[3] = mirror ? -d3 : d3;
}

// Rows of the tables, 32 floats (128 bytes) per slot: point j of axis a at
// [10 a + 2 j]: value and first derivative in SplineTable::lo, second and
// third derivative in SplineTable::hi (entries 30 and 31 unused).
constexpr int SPL_ROW = 32;

__device__ __forceinline__ float2 spl(const float* row, int axis, int j)
{
   return reinterpret_cast<const float2*>(row)[5 * axis + j];
}

// one axis of one slot: origin (wrapped into the grid) and the 5 x 4 weights
__device__ __forceinline__ int spline_axis(float x, float rbox, int nfft, int axis, float* __restrict__ lo,
   float* __restrict__ hi)
{
   float w = x * rbox;
   w = w + 0.5f - floorf(w + 0.5f);
   const float fr = nfft * w;
   int i = (int)floorf(fr);
   w = fr - i;
   i -= BSORDER - 1;
   i += (i < 0 ? nfft : 0);
   float th[5][4];
   spline_piece<0>(w, th[0]);
   spline_piece<1>(w, th[1]);
   spline_piece<2>(w, th[2]);
   spline_piece<3>(w, th[3]);
   spline_piece<4>(w, th[4]);
   float2* l = reinterpret_cast<float2*>(lo) + 5 * axis;
   float2* h = reinterpret_cast<float2*>(hi) + 5 * axis;
#pragma unroll
   for (int j = 0; j < 5; ++j) {
      l[j] = make_float2(th[j][0], th[j][1]);
      h[j] = make_float2(th[j][2], th[j][3]);
   }
   return i;
}

}  // namespace t9gb
