// Order-5 B-splines of the PME sites: the table of every slot's grid origin,
// spline values and derivatives, formed once per position update
// (k_scatter_pos) and read by the spread and gather kernels (pme.cu).
// Weights as bsplgen (include/seq/bsplgen.h:27-116), grid origins as
// src/cu/pme.cu:31-58.
#pragma once
#include "common.cuh"

namespace t9gb {

// weights and derivatives of the five points of one axis at fraction w
template <int LEVEL>
__device__ __forceinline__ void bspline5(float w, float th[5][LEVEL])
{
   float b[6][6];  // b[order][i], 1-based
   b[2][2] = w;
   b[2][1] = 1.f - w;
   b[3][3] = 0.5f * w * b[2][2];
   b[3][2] = 0.5f * ((1.f + w) * b[2][1] + (2.f - w) * b[2][2]);
   b[3][1] = 0.5f * (1.f - w) * b[2][1];
#pragma unroll
   for (int i = 4; i <= 5; ++i) {
      const int k = i - 1;
      const float denom = 1.f / k;
      b[i][i] = denom * w * b[k][k];
#pragma unroll
      for (int j = 1; j <= i - 2; ++j)
         b[i][i - j] = denom * ((w + j) * b[k][i - j - 1] + (i - j - w) * b[k][i - j]);
      b[i][1] = denom * (1.f - w) * b[k][1];
   }
   // derivative rows by repeated differencing of the lower-order rows
#pragma unroll
   for (int lv = 2; lv <= LEVEL; ++lv) {
      const int k = 5 - lv + 1;
#pragma unroll
      for (int pass = 0; pass < lv - 1; ++pass) {
         const int top = 5 - (lv - 2) + pass;
         b[k][top] = b[k][top - 1];
#pragma unroll
         for (int i = top - 1; i >= 2; --i)
            b[k][i] = b[k][i - 1] - b[k][i];
         b[k][1] = -b[k][1];
      }
   }
#pragma unroll
   for (int i = 1; i <= 5; ++i)
#pragma unroll
      for (int j = 1; j <= LEVEL; ++j)
         th[i - 1][j - 1] = b[5 - j + 1][i];
}

// Rows of the tables, 32 floats (128 bytes) per slot: point j of axis a at
// [10 a + 2 j]: value and first derivative in PmeGrid::spl_lo, second and
// third derivative in PmeGrid::spl_hi (entries 30 and 31 unused).
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
   bspline5<4>(w, th);
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
