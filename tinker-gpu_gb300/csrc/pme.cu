// PME reciprocal-space field for AMOEBA: B-spline spreading of fractional
// multipoles or induced dipoles, convolution with the Ewald influence
// function, and the gather of potential derivatives fused with the
// reciprocal-self field terms.
//
// Reference pieces replaced (src/cu/pme.cu): gridPut_cu1<MPOLE> :14-183,
// gridPut_cu2<UIND> :185-255, fphiGet_cu<MPOLE/UIND2> :383-870, pmeConv_cu1
// :908-1031, cmpToFmp/cuindToFuind/fphiToCphi :1052-1300, and the recip-self
// kernels dfieldEwaldRecipSelfP2_cu1 / ufieldEwaldRecipSelfP1_cu1
// (src/cu/amoeba/field.cu:12-33, :71-118).
//
// Differences by design (same results up to rounding):
//  - the fractional transforms are folded into spread and gather (orthogonal
//    boxes: the transforms are diagonal);
//  - dfield and ufield only consume first derivatives of the potential, so the
//    gather evaluates 3 (MPOLE) or 6 (UIND) sums instead of 20 / 20;
//  - the influence function exp(-pi^2 h^2/a^2)/(pi V h^2 |b|^2) is tabulated
//    once per box (the reference recomputes it in every pmeConv call);
//  - the grid accumulates in 64-bit fixed point (order-independent), then one
//    pass converts it to the complex float grid and clears the fixed grid.
#include <cmath>
#include <utility>
#include <vector>

#include "common.cuh"
#include "reduce.cuh"
#include "spline.cuh"

namespace t9gb {

// ---------------------------------------------------------------------------
// B-spline moduli |b(m)|^2 (Essmann et al., J. Chem. Phys. 103, 8577 (1995))
// with Tinker's optimal-zeta correction of Euler-spline zeros.

static void cardinal_bspline_knots(int order, double* c)
{
   const double x = 0;
   c[0] = 1 - x;
   c[1] = x;
   for (int k = 3; k <= order; ++k) {
      double denom = 1.0 / (k - 1);
      c[k - 1] = x * c[k - 2] * denom;
      for (int i = 1; i <= k - 2; ++i)
         c[k - i - 1] = ((x + i) * c[k - i - 2] + (k - i - x) * c[k - i - 1]) * denom;
      c[0] = (1 - x) * c[0] * denom;
   }
}

static void bspline_moduli(int nfft, int order, std::vector<double>& mod)
{
   const double pi = 3.14159265358979323846;
   std::vector<double> arr(nfft + order + 2, 0.0);
   double c[16];
   cardinal_bspline_knots(order, c);
   for (int i = 0; i < order; ++i)
      arr[i + 1] = c[i];
   mod.assign(nfft, 0.0);
   for (int i = 0; i < nfft; ++i) {
      double s1 = 0, s2 = 0;
      for (int j = 0; j < nfft; ++j) {
         double arg = 2 * pi * (double)i * (double)j / nfft;
         s1 += arr[j] * std::cos(arg);
         s2 += arr[j] * std::sin(arg);
      }
      mod[i] = s1 * s1 + s2 * s2;
   }
   const double eps = 1.0e-7;
   if (mod[0] < eps)
      mod[0] = 0.5 * mod[1];
   for (int i = 1; i < nfft - 1; ++i)
      if (mod[i] < eps)
         mod[i] = 0.5 * (mod[i - 1] + mod[i + 1]);
   if (mod[nfft - 1] < eps)
      mod[nfft - 1] = 0.5 * mod[nfft - 2];
   for (int i = 0; i < nfft; ++i) {
      int k = (i + 1 > nfft / 2) ? i - nfft : i;
      double zeta = 1;
      if (k != 0) {
         double s1 = 1, s2 = 1, f = pi * k / nfft;
         for (int j = 1; j <= 50; ++j) {
            double a1 = f / (f + pi * j), a2 = f / (f - pi * j);
            s1 += std::pow(a1, order) + std::pow(a2, order);
            s2 += std::pow(a1, 2 * order) + std::pow(a2, 2 * order);
         }
         zeta = s2 / s1;
      }
      mod[i] *= zeta * zeta;
   }
}

struct GridParams {
   int n1, n2, n3;
   float r1, r2, r3;  // 1/box
   float a1, a2, a3;  // nfft / box
   float selfterm;    // 4 a^3 / (3 sqrt(pi))
   float pk_s, pk_lim;  // dipole grids: 32-bit fixed-point scale, per-contribution guard
   int* range;          // set when a contribution reaches pk_lim
};

__device__ __forceinline__ void site(const GridParams& G, float4 p, int& i1, int& i2, int& i3, float& w1, float& w2,
   float& w3)
{
   float w = p.x * G.r1;
   w = w + 0.5f - floorf(w + 0.5f);
   float fr = G.n1 * w;
   i1 = (int)floorf(fr);
   w1 = fr - i1;
   w = p.y * G.r2;
   w = w + 0.5f - floorf(w + 0.5f);
   fr = G.n2 * w;
   i2 = (int)floorf(fr);
   w2 = fr - i2;
   w = p.z * G.r3;
   w = w + 0.5f - floorf(w + 0.5f);
   fr = G.n3 * w;
   i3 = (int)floorf(fr);
   w3 = fr - i3;
   i1 -= BSORDER - 1;
   i2 -= BSORDER - 1;
   i3 -= BSORDER - 1;
   i1 += (i1 < 0 ? G.n1 : 0);
   i2 += (i2 < 0 ? G.n2 : 0);
   i3 += (i3 < 0 ? G.n3 : 0);
}

// Fixed-point grid: one 64-bit word per point.  Multipole grids hold the
// real part at scale 2^40 (to_fx).  Dipole grids pack the d value (high 32
// bits) and the p value (low 32 bits) as 32-bit fixed point at scale pk_s
// (2^24, or 2^16 after a range fallback): the word sum is A 2^32 + B for the
// sums A, B of the halves, and both are recovered exactly while each stays
// within the signed 32-bit range, so one reduction carries both grids.

// fire-and-forget 64-bit reduction (no value returned, so the warp does not
// wait on it)
__device__ __forceinline__ void red_u64(unsigned long long* q, size_t idx, unsigned long long v)
{
   asm volatile("red.global.add.u64 [%0], %1;" ::"l"(q + idx), "l"(v) : "memory");
}

__device__ __forceinline__ void grid_add(unsigned long long* q, size_t idx, float v)
{
   if (v != 0.f)
      red_u64(q, idx, (unsigned long long)to_fx(v));
}

// d and p values of one point into one word; false when a value is at or
// above pk_lim in magnitude (1/32 of the half's range) or not a number: the
// caller raises the range flag, and the grid's user solves again
__device__ __forceinline__ bool grid_add2(unsigned long long* q, float vd, float vp, const GridParams& G)
{
   const bool ok = (fabsf(vd) < G.pk_lim) & (fabsf(vp) < G.pk_lim);
   const long long a = __float2int_rn(vd * G.pk_s), b = __float2int_rn(vp * G.pk_s);
   red_u64(q, 0, (unsigned long long)(a * 4294967296ll + b));
   return ok;
}

// one word of the fixed-point grid as a complex value
__device__ __forceinline__ float2 grid_word(long long w, int packed, float inv)
{
   if (!packed)
      return make_float2(from_fx(w), 0.f);
   const int b = (int)(unsigned)(unsigned long long)w;
   const int a = (int)((w - (long long)b) >> 32);
   return make_float2((float)a * inv, (float)b * inv);
}

// the guard on the sums of a packed word: each contribution stays below
// 2^26, so a half at or above 2^30 in magnitude (16 or more near-limit
// contributions of one sign, far beyond real grids) is taken as a sum that
// may have left the 32-bit range, and the solve is repeated at the wider
// scale, as for a large contribution
__device__ __forceinline__ bool grid_word_big(long long w, int packed)
{
   if (!packed)
      return false;
   const int b = (int)(unsigned)(unsigned long long)w;
   const int a = (int)((w - (long long)b) >> 32);
   return a >= (1 << 30) || a <= -(1 << 30) || b >= (1 << 30) || b <= -(1 << 30);
}

// The sites' spline tables and grid origins (spline.cuh) as the kernels take
// them.
struct Sites {
   const int4* org;
   const float *lo, *hi;
};

// Byte stride between z planes of a grid of 8-byte points.
__device__ __forceinline__ unsigned plane_bytes(const GridParams& G) { return 8u * (unsigned)G.n1 * (unsigned)G.n2; }

// Byte offset within a plane of point (ix, jy) of a site's support.
__device__ __forceinline__ unsigned column_bytes(const GridParams& G, int4 o, int ix, int jy)
{
   int xb = o.x + ix;
   xb -= (xb >= G.n1 ? G.n1 : 0);
   int yb = o.y + jy;
   yb -= (yb >= G.n2 ? G.n2 : 0);
   return 8u * ((unsigned)yb * (unsigned)G.n1 + (unsigned)xb);
}

// a b + c d with the product c d rounded: the roundings of a grid value are
// written out, so that they do not depend on how a kernel is laid out
__device__ __forceinline__ float dot2(float a, float b, float c, float d)
{
   return __fmaf_rn(a, b, __fmul_rn(c, d));
}

// Spreading, one warp per atom: lane (ix, jy) < 25 owns one column of five z
// points, so that each of a warp's five reductions covers five rows of five
// consecutive words.  MODE 0 spreads fractional multipoles into the real
// part; MODE 1 spreads fractional d dipoles into the real and p dipoles into
// the imaginary part.  rp rows are 12 floats (q, d, quadrupole, ...), u rows
// 8.  DIR (MODE 1): the dipoles are the CG search direction p = z + b p_old
// (src = p_old, z8 = z, b from scal), formed as each row is read; dir8 (may
// be null, else = src): p is stored there, each row by the one warp that
// reads it.
template <int MODE, bool DIR = false>
__global__ void __launch_bounds__(256) k_spread(int n, GridParams G, Sites S, const float* src,
   const float* __restrict__ z8, const double* __restrict__ scal, unsigned long long* __restrict__ q, float* dir8)
{
   // the sites do not depend on the programmatic predecessor: they are read
   // before the wait for it (no-op otherwise)
   const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const int lane = threadIdx.x & 31;
   if (s >= n || lane >= 25)
      return;
   const int ix = lane % 5, jy = lane / 5;
   const int4 o = S.org[s];
   const float* lo = S.lo + (size_t)SPL_ROW * s;
   const float* hi = S.hi + (size_t)SPL_ROW * s;
   const float2 tx = spl(lo, 0, ix), ty = spl(lo, 1, jy);
   float2 tz[5];
#pragma unroll
   for (int k = 0; k < 5; ++k)
      tz[k] = spl(lo, 2, k);
   char* col = reinterpret_cast<char*>(q) + column_bytes(G, o, ix, jy);
   const unsigned plane = plane_bytes(G);
   const float u0 = ty.x, u1 = ty.y;
   if (MODE == 0) {
      const float x2 = spl(hi, 0, ix).x, u2 = spl(hi, 1, jy).x;
      float z2[5];
#pragma unroll
      for (int k = 0; k < 5; ++k)
         z2[k] = spl(hi, 2, k).x;
      pdl_wait();
      pdl_trigger();
      const float* m = src + 12 * s;
      // Cartesian -> fractional (orthogonal box; quadrupole off-diagonals doubled)
      const float f0 = m[0];
      const float fx = G.a1 * m[1], fy = G.a2 * m[2], fz = G.a3 * m[3];
      const float fxx = G.a1 * G.a1 * m[4], fyy = G.a2 * G.a2 * m[5], fzz = G.a3 * G.a3 * m[6];
      const float fxy = 2.f * G.a1 * G.a2 * m[7], fxz = 2.f * G.a1 * G.a3 * m[8], fyz = 2.f * G.a2 * G.a3 * m[9];
#pragma unroll
      for (int kz = 0; kz < 5; ++kz) {
         int zb = o.z + kz;
         zb -= (zb >= G.n3 ? G.n3 : 0);
         const float v0 = tz[kz].x, v1 = tz[kz].y, v2 = z2[kz];
         float term0 = dot2(f0 * u0, v0, fy * u1, v0);
         term0 = __fmaf_rn(fz * u0, v1, term0);
         term0 = __fmaf_rn(fyy * u2, v0, term0);
         term0 = __fmaf_rn(fzz * u0, v2, term0);
         term0 = __fmaf_rn(fyz * u1, v1, term0);
         const float term1 = __fmaf_rn(fxz * u0, v1, dot2(fx * u0, v0, fxy * u1, v0));
         const float term2 = fxx * u0 * v0;
         grid_add(reinterpret_cast<unsigned long long*>(col + (size_t)(unsigned)zb * plane), 0,
            __fmaf_rn(term2, x2, dot2(term0, tx.x, term1, tx.y)));
      }
   } else {
      pdl_wait();
      pdl_trigger();
      float u[8];
      if (DIR) {
         dir_row(src, z8, s, (float)scal[S_B_D], (float)scal[S_B_P], u);
         if (dir8) {
            __syncwarp(0x1ffffff);  // every lane has read the row
            float v = u[0];
#pragma unroll
            for (int c = 1; c < 6; ++c)
               if (lane == c)
                  v = u[c];
            if (lane < 6)
               dir8[8 * s + lane] = v;
         }
      } else {
         load8(src, s, u);
      }
      const float dx = G.a1 * u[0], dy = G.a2 * u[1], dz = G.a3 * u[2];
      const float px = G.a1 * u[3], py = G.a2 * u[4], pz = G.a3 * u[5];
      bool ok = true;
#pragma unroll
      for (int kz = 0; kz < 5; ++kz) {
         int zb = o.z + kz;
         zb -= (zb >= G.n3 ? G.n3 : 0);
         const float v0 = tz[kz].x, v1 = tz[kz].y;
         const float d01 = dot2(dy * u1, v0, dz * u0, v1), d11 = dx * u0 * v0;
         const float p01 = dot2(py * u1, v0, pz * u0, v1), p11 = px * u0 * v0;
         ok &= grid_add2(reinterpret_cast<unsigned long long*>(col + (size_t)(unsigned)zb * plane),
            dot2(d01, tx.x, d11, tx.y), dot2(p01, tx.x, p11, tx.y), G);
      }
      if (!ok)
         atomicOr(G.range, 1);
   }
}

// fixed -> complex float, clearing the fixed grid for the next spread
__global__ void k_fx_to_grid(size_t ng, long long* __restrict__ q, float2* __restrict__ g, int packed, float inv,
   int* __restrict__ range)
{
   bool big = false;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ng; i += (size_t)gridDim.x * blockDim.x) {
      const long long w = q[i];
      big |= grid_word_big(w, packed);
      g[i] = grid_word(w, packed, inv);
      q[i] = 0;
   }
   if (big)
      atomicOr(range, 1);
}

// reciprocal convolution with the tabulated influence function
__global__ void k_conv(size_t ng, const float* __restrict__ infl, float2* __restrict__ g)
{
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ng; i += (size_t)gridDim.x * blockDim.x) {
      float2 v = g[i];
      float f = infl[i];
      g[i] = make_float2(v.x * f, v.y * f);
   }
}

// Gather of the first potential derivatives fused with the recip + self
// field, one warp per atom.  The points are loaded as lane (ix, jy) < 25
// taking a column of five z points, so that each of a warp's five loads
// covers five rows of five consecutive points (about six 128-byte lines; a
// lane per row touches 25 lines in each load and was bound by them), then
// exchanged through shared memory: lane (jy, kz) sums one row of five x
// points, and a fixed xor tree combines the rows (warp_sums).  MODE 0:
// real part -> d and p field, self term with the permanent dipole.  MODE 1:
// real -> d, imaginary -> p, self term with the induced dipoles.  Plain
// stores, rows of 8 floats.
// AP (MODE 1, ACC): the dipoles are the CG search direction p = z + b p_old
// (P.conj = p_old, P.zrsd = z); instead of the field, the lanes that hold
// the components store p and Ap = p/alpha - field, and the block partials of
// p.Ap give, in the last block, the step length a = s / p.Ap.  Atoms are
// visited warp-strided over at most RED_MAX blocks.
// LATE: the kernel has not waited for its programmatic predecessor yet; the
// site's splines are read first, then the wait, then the grid and dipole
// reads, so the prologue overlaps the predecessor.
template <int MODE, bool ACC, bool AP, bool DIR, bool LATE = false>
__device__ __forceinline__ void gather_atom(int s, int lane, const GridParams& G, const Sites& S,
   const float2* __restrict__ g, const float* __restrict__ rp, const float* __restrict__ u8, float* __restrict__ out,
   const PcgAp& P, float bd, float bp, float* pap, float2* xch)
{
   constexpr int NC = MODE == 1 ? 6 : 3;
   float acc[NC];
#pragma unroll
   for (int c = 0; c < NC; ++c)
      acc[c] = 0.f;
   const int4 o = S.org[s];
   const float* lo = S.lo + (size_t)SPL_ROW * s;
   const int q5 = lane % 5, d5 = lane / 5;  // (ix, jy) loading, (jy, kz) summing
   float2 tx[5], ty, tz;
   if (lane < 25) {
#pragma unroll
      for (int k = 0; k < 5; ++k)
         tx[k] = spl(lo, 0, k);
      ty = spl(lo, 1, q5);
      tz = spl(lo, 2, d5);
   }
   if (LATE)
      pdl_wait();
   float* xr = reinterpret_cast<float*>(xch);
   if (lane < 25) {
      const unsigned plane = plane_bytes(G);
      const char* col = reinterpret_cast<const char*>(g) + column_bytes(G, o, q5, d5);
      float2 q[5];
#pragma unroll
      for (int kz = 0; kz < 5; ++kz) {
         int zb = o.z + kz;
         zb -= (zb >= G.n3 ? G.n3 : 0);
         const float2* p = reinterpret_cast<const float2*>(col + (size_t)(unsigned)zb * plane);
         if (MODE == 1)
            q[kz] = *p;
         else
            q[kz].x = p->x;
      }
#pragma unroll
      for (int kz = 0; kz < 5; ++kz)
         if (MODE == 1)
            xch[25 * kz + lane] = q[kz];
         else
            xr[25 * kz + lane] = q[kz].x;
   }
   __syncwarp();
   if (lane < 25) {
      // row (jy, kz) = 5 lane .. 5 lane + 4 of the exchanged points
      float rt0 = 0.f, rt1 = 0.f, it0 = 0.f, it1 = 0.f;
#pragma unroll
      for (int ix = 0; ix < 5; ++ix) {
         float2 qv;
         if (MODE == 1)
            qv = xch[5 * lane + ix];
         else
            qv.x = xr[5 * lane + ix];
         rt0 += qv.x * tx[ix].x;
         rt1 += qv.x * tx[ix].y;
         if (MODE == 1) {
            it0 += qv.y * tx[ix].x;
            it1 += qv.y * tx[ix].y;
         }
      }
      const float u0 = ty.x, u1 = ty.y, v0 = tz.x, v1 = tz.y;
      acc[0] = rt1 * u0 * v0;
      acc[1] = rt0 * u1 * v0;
      acc[2] = rt0 * u0 * v1;
      if (MODE == 1) {
         acc[NC - 3] = it1 * u0 * v0;
         acc[NC - 2] = it0 * u1 * v0;
         acc[NC - 1] = it0 * u0 * v1;
      }
   }
   __syncwarp();  // the exchange buffer is free for the warp's next atom
   const float sum = warp_sums<NC>(acc, lane);
   const int c = sum_slot<NC>(lane);
   if (c < 0)
      return;
   // the lane that holds component c finishes it
   const int d = c < 3 ? c : c - 3, x = 8 * s + c;
   const float gc = d == 0 ? G.a1 : (d == 1 ? G.a2 : G.a3);
   if (AP) {
      // p, its recip + self field added to the real-space field, Ap =
      // p/alpha - field, and p.Ap
      const float p = __fmaf_rn(c < 3 ? bd : bp, P.conj[x], P.zrsd[x]);
      const float fld = out[x] + (G.selfterm * p - gc * sum);
      const float v = P.polinv[s] * p - fld;
      P.vec[x] = v;
      P.conj[x] = p;
      pap[c < 3 ? 0 : 1] += p * v;
      return;
   }
   if (MODE == 0) {
      const float r = -gc * sum + G.selfterm * rp[12 * s + 1 + d];
      out[x] = ACC ? out[x] + r : r;
      out[x + 3] = ACC ? out[x + 3] + r : r;
      return;
   }
   const float u = DIR ? __fmaf_rn(c < 3 ? bd : bp, P.conj[x], P.zrsd[x]) : u8[x];
   const float r = G.selfterm * u - gc * sum;
   // ACC: add to the real-space field already stored (the same two-operand
   // sum the real-space kernel forms when it adds this result as its base)
   out[x] = ACC ? out[x] + r : r;
}

template <int MODE, bool ACC, bool AP = false, bool DIR = false>
__global__ void __launch_bounds__(256, 6) k_gather_field(int n, GridParams G, Sites S,
   const float2* __restrict__ g, const float* __restrict__ rp, const float* __restrict__ u8, float* __restrict__ out,
   PcgAp P)
{
   // the plain gather waits inside gather_atom, after its position-only prologue
   constexpr bool LATE = !AP && !DIR;
   __shared__ float2 xch[8][125];
   if (!LATE)
      pdl_wait();
   const int lane = threadIdx.x & 31;
   if (!AP) {
      const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
      float bd = 0.f, bp = 0.f;
      if (DIR) {
         bd = (float)P.scal[S_B_D];
         bp = (float)P.scal[S_B_P];
      }
      if (s < n)
         gather_atom<MODE, ACC, false, DIR, LATE>(s, lane, G, S, g, rp, u8, out, P, bd, bp, nullptr, xch[threadIdx.x >> 5]);
      else if (LATE)
         pdl_wait();
      return;
   }
   __shared__ double sh[64];
   const float bd = (float)P.scal[S_B_D], bp = (float)P.scal[S_B_P];
   float pap[2] = {0.f, 0.f};
   const int nw = (gridDim.x * blockDim.x) >> 5;
   for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < n; s += nw)
      gather_atom<MODE, ACC, true, false>(s, lane, G, S, g, rp, u8, out, P, bd, bp, pap, xch[threadIdx.x >> 5]);
   store_partials_f<2>(P.red, R_PAP_D, pap, sh);
   if (!last_block(P.state + ST_TICKET1))
      return;
   double tot[2];
   sum_slots(P.red, R_PAP_D, 2, gridDim.x, sh, tot);
   if (threadIdx.x == 0) {  // the step lengths in FP32 (used as FP32)
      P.scal[S_A_D] = tot[0] == 0 ? 0.0 : (double)((float)P.scal[S_SUM_D] / (float)tot[0]);
      P.scal[S_A_P] = tot[1] == 0 ? 0.0 : (double)((float)P.scal[S_SUM_P] / (float)tot[1]);
   }
}

// Multipole reciprocal + self energy per atom (warp per atom, level-3
// weights): e = 1/2 f sum_k fmp_k fphi_k (src/cu/hippo/empole.cu:202-335)
// and the Ewald self energy (include/seq/emselfamoeba.h:7-37), stored per
// atom in e_atom[s] and e_self[s].
__global__ void __launch_bounds__(256) k_empole_recip_self(int n, GridParams G, float f, float aewald,
   const float4* __restrict__ spos, const float2* __restrict__ g, const float* __restrict__ rp,
   double* __restrict__ e_atom, double* __restrict__ e_self)
{
   const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const int lane = threadIdx.x & 31;
   if (s >= n)
      return;
   int i1, i2, i3;
   float w1, w2, w3;
   site(G, spos[s], i1, i2, i3, w1, w2, w3);
   float phi[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
   if (lane < 25) {
      float t1[5][3], t2[5][3], t3[5][3];
      bspline5<3>(w1, t1);
      bspline5<3>(w2, t2);
      bspline5<3>(w3, t3);
      const int jy = lane % 5, kz = lane / 5;
      int zb = i3 + kz;
      zb -= (zb >= G.n3 ? G.n3 : 0);
      int yb = i2 + jy;
      yb -= (yb >= G.n2 ? G.n2 : 0);
      const size_t row = ((size_t)zb * G.n2 + yb) * G.n1;
      float t0 = 0.f, ta = 0.f, tb = 0.f;
#pragma unroll
      for (int ix = 0; ix < 5; ++ix) {
         int xb = i1 + ix;
         xb -= (xb >= G.n1 ? G.n1 : 0);
         const float q = g[row + xb].x;
         t0 += q * t1[ix][0];
         ta += q * t1[ix][1];
         tb += q * t1[ix][2];
      }
      const float u0 = t2[jy][0], u1 = t2[jy][1], u2 = t2[jy][2];
      const float v0 = t3[kz][0], v1 = t3[kz][1], v2 = t3[kz][2];
      phi[0] = t0 * u0 * v0;
      phi[1] = ta * u0 * v0;
      phi[2] = t0 * u1 * v0;
      phi[3] = t0 * u0 * v1;
      phi[4] = tb * u0 * v0;
      phi[5] = t0 * u2 * v0;
      phi[6] = t0 * u0 * v2;
      phi[7] = ta * u1 * v0;
      phi[8] = ta * u0 * v1;
      phi[9] = t0 * u1 * v1;
   }
#pragma unroll
   for (int c = 0; c < 10; ++c)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
         phi[c] += __shfl_xor_sync(0xffffffffu, phi[c], o);
   if (lane != 0)
      return;
   const float* m = rp + 12 * s;
   const double fmp[10] = {m[0], G.a1 * m[1], G.a2 * m[2], G.a3 * m[3], G.a1 * G.a1 * m[4], G.a2 * G.a2 * m[5],
      G.a3 * G.a3 * m[6], 2.f * G.a1 * G.a2 * m[7], 2.f * G.a1 * G.a3 * m[8], 2.f * G.a2 * G.a3 * m[9]};
   double e = 0;
   for (int c = 0; c < 10; ++c)
      e += fmp[c] * (double)phi[c];
   e_atom[s] = 0.5 * f * e;
   const double a2 = 2.0 * aewald * aewald;
   const double fterm = -(double)f * aewald / 1.77245385090551602730;
   const double cii = (double)m[0] * m[0];
   const double dii = (double)m[1] * m[1] + (double)m[2] * m[2] + (double)m[3] * m[3];
   const double qii = 2.0 * ((double)m[7] * m[7] + (double)m[8] * m[8] + (double)m[9] * m[9]) + (double)m[4] * m[4]
      + (double)m[5] * m[5] + (double)m[6] * m[6];
   e_self[s] = fterm * (cii + a2 * (dii / 3.0 + 2.0 * a2 * qii * 0.2));
}

// ---------------------------------------------------------------------------
// Fused 3-D FFT + convolution for cubic power-of-two grids (N = 32, 64, 128
// points per edge), replacing cuFFT's six kernels plus the fixed-point
// conversion and the convolution of one pass by three kernels:
//   k_fft_plane<FROM_FX, forward>: fixed-point grid -> float (the fixed-point
//     grid is cleared for the next spread), 2-D forward FFT of each z plane;
//   k_fft_zline<MODE 2>: forward FFT along z, times the influence function,
//     inverse FFT along z, for 16 x-adjacent lines per block (the virial path
//     splits it into MODE 0 forward / MODE 1 inverse around the k-space pass);
//   k_fft_plane<inverse>: 2-D inverse FFT of each plane.
// A line transform of N = N1 x T points runs on T threads (8; 4 for N = 32)
// of one warp, each holding N1 points in registers: an N1-point DFT over the
// stride-T subsequence, the twiddle W_N^(t k1), an exchange through shared
// memory, then N1 / T T-point DFTs per thread (Cooley-Tukey with
// n = n1 T + n2, k = k1 + N1 k2).  Forward e^{-2 pi i k n / N}, inverse
// unnormalised, as cuFFT's C2C; the twiddles come from a table computed in
// double precision.

__constant__ float2 c_tw[128];  // e^{-2 pi i k / 128}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
   return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__host__ __device__ constexpr int brev_c(int x, int bits)
{
   int r = 0;
   for (int b = 0; b < bits; ++b) {
      r = (r << 1) | (x & 1);
      x >>= 1;
   }
   return r;
}

__host__ __device__ constexpr int log2_c(int m) { return m <= 1 ? 0 : 1 + log2_c(m / 2); }

// in-register M-point DFT (M = 4, 8, 16), natural order in and out;
// tw: e^{-2 pi i k / 128} in shared memory (uniform indices: broadcasts)
template <int M, bool INV>
__device__ __forceinline__ void dft_reg(float2* v, const float2* tw)
{
   constexpr int L = log2_c(M);
#pragma unroll
   for (int i = 0; i < M; ++i) {
      const int j = brev_c(i, L);
      if (j > i) {
         const float2 a = v[i];
         v[i] = v[j];
         v[j] = a;
      }
   }
#pragma unroll
   for (int st = 1; st <= L; ++st) {
      const int len = 1 << st, half = len / 2, step = 128 / len;
#pragma unroll
      for (int b = 0; b < M; b += len)
#pragma unroll
         for (int k = 0; k < half; ++k) {
            float2 w = tw[k * step];
            if (INV)
               w.y = -w.y;
            const float2 a = v[b + k];
            const float2 c = k == 0 ? v[b + k + half] : cmulf(w, v[b + k + half]);
            v[b + k] = make_float2(a.x + c.x, a.y + c.y);
            v[b + k + half] = make_float2(a.x - c.x, a.y - c.y);
         }
   }
}

// Shared-memory swizzle of a line index: the low bits within each block of T
// are XORed with the block number (and the block group), so the strided
// step-2 reads of fft_line and the column passes spread over the banks.
template <int T>
__device__ __forceinline__ int fsig(int i)
{
   return i ^ (((i / T) + (i / (T * T))) & (T - 1));
}

// One N-point line, element i at line[fsig(i) * ls], transformed in place by
// the T threads t = 0..T-1 of one warp (every thread of the warp takes part
// in some line).
// wt[k1] = W_N^(t k1) for this thread's t, read once per kernel from the
// table (its thread-dependent indices would conflict on every line).
template <int N, int T>
__device__ __forceinline__ void fft_twiddles(int t, const float2* tw, float2* wt)
{
   if (N / T <= 8) {
#pragma unroll
      for (int k1 = 0; k1 < N / T; ++k1)
         wt[k1] = tw[((t * k1) & (N - 1)) * (128 / N)];
   }
}

template <int N, int T, bool INV>
__device__ __forceinline__ void fft_line(float2* line, int ls, int t, const float2* tw, const float2* wt)
{
   constexpr int N1 = N / T, J = N1 / T;
   float2 v[N1];
#pragma unroll
   for (int n1 = 0; n1 < N1; ++n1)
      v[n1] = line[fsig<T>(n1 * T + t) * ls];
   dft_reg<N1, INV>(v, tw);
#pragma unroll
   for (int k1 = 1; k1 < N1; ++k1) {
      // registers for up to 8 twiddles; the 128-point lines (1024-thread
      // planes) read the table rather than spill
      float2 w = N1 <= 8 ? wt[k1] : tw[((t * k1) & (N - 1)) * (128 / N)];
      if (INV)
         w.y = -w.y;
      v[k1] = cmulf(v[k1], w);
   }
   __syncwarp();
#pragma unroll
   for (int k1 = 0; k1 < N1; ++k1)
      line[fsig<T>(k1 * T + t) * ls] = v[k1];
   __syncwarp();
   float2 u[J][T];
#pragma unroll
   for (int j = 0; j < J; ++j) {
      const int k1 = t * J + j;
#pragma unroll
      for (int n2 = 0; n2 < T; ++n2)
         u[j][n2] = line[fsig<T>(k1 * T + n2) * ls];
      dft_reg<T, INV>(u[j], tw);
   }
   __syncwarp();
#pragma unroll
   for (int j = 0; j < J; ++j)
#pragma unroll
      for (int k2 = 0; k2 < T; ++k2)
         line[fsig<T>(t * J + j + N1 * k2) * ls] = u[j][k2];
   __syncwarp();
}

template <int N>
__host__ __device__ constexpr int fft_threads_per_line()
{
   return N == 32 ? 4 : 8;
}

// row pitch of the plane (float2) and of the z-line tile
template <int N>
__host__ __device__ constexpr int fft_plane_ld()
{
   return N == 32 ? N + 4 : N + 2;
}

template <int N>
__host__ __device__ constexpr int fft_zline_ld()
{
   return N == 32 ? 20 : 18;
}

// 2-D FFT (x then y) of z plane blockIdx.x; N * T threads, dynamic shared
// memory N (N + 1) + 128 float2
template <int N, bool FROM_FX, bool INV>
__global__ void __launch_bounds__(N * fft_threads_per_line<N>()) k_fft_plane(long long* __restrict__ qfx,
   float2* __restrict__ g, int packed, float inv, int* __restrict__ range)
{
   pdl_wait();
   pdl_trigger();  // the next kernel may stage its blocks and run its prologue
   // element (y, x) at fsm[fsig(y) LD + fsig(x)]; the padding keeps the two
   // lines of a 16-thread shared-memory phase on different banks
   constexpr int T = fft_threads_per_line<N>(), LD = fft_plane_ld<N>(), NT = N * T, R = N / T;
   extern __shared__ float2 fsm[];
   float2* tw = fsm + N * LD;
   for (int k = threadIdx.x; k < 128; k += NT)
      tw[k] = c_tw[k];
   const size_t base = (size_t)blockIdx.x * N * N;
   // element e = threadIdx.x + r NT, r < R: all loads of a chunk in flight together
   bool big = false;
#pragma unroll
   for (int c = 0; c < R; c += 8) {
      float2 v[8];
      if (FROM_FX) {
         long long* q = qfx + base + threadIdx.x;
         long long f[8];
#pragma unroll
         for (int r = 0; r < 8; ++r)
            f[r] = q[(c + r) * NT];
#pragma unroll
         for (int r = 0; r < 8; ++r) {
            q[(c + r) * NT] = 0;
            big |= grid_word_big(f[r], packed);
            v[r] = grid_word(f[r], packed, inv);
         }
      } else {
#pragma unroll
         for (int r = 0; r < 8; ++r)
            v[r] = g[base + threadIdx.x + (c + r) * NT];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
         const int e = threadIdx.x + (c + r) * NT;
         fsm[fsig<T>(e / N) * LD + fsig<T>(e % N)] = v[r];
      }
   }
   if (FROM_FX && big)
      atomicOr(range, 1);
   __syncthreads();
   const int line = threadIdx.x / T, t = threadIdx.x % T;
   float2 wt[N / T];
   fft_twiddles<N, T>(t, tw, wt);
   fft_line<N, T, INV>(fsm + fsig<T>(line) * LD, 1, t, tw, wt);  // row y = line, along x
   __syncthreads();
   fft_line<N, T, INV>(fsm + fsig<T>(line), LD, t, tw, wt);  // column x = line, along y
   __syncthreads();
#pragma unroll
   for (int r = 0; r < R; ++r) {
      const int e = threadIdx.x + r * NT;
      g[base + e] = fsm[fsig<T>(e / N) * LD + fsig<T>(e % N)];
   }
}

// Lines along z of 16 adjacent x at one y.  MODE 0 forward, 1 inverse,
// 2 forward, influence function, inverse.
template <int N, int MODE>
__global__ void __launch_bounds__(16 * fft_threads_per_line<N>()) k_fft_zline(const float* __restrict__ infl,
   float2* __restrict__ g)
{
   pdl_wait();
   pdl_trigger();  // the next kernel may stage its blocks and run its prologue
   // element z of line l at sm[fsig(z) LD + l]
   constexpr int T = fft_threads_per_line<N>(), XL = 16, LD = fft_zline_ld<N>(), NT = XL * T, R = N / T;
   __shared__ float2 sm[N * LD];
   __shared__ float2 tw[128];
   for (int k = threadIdx.x; k < 128; k += NT)
      tw[k] = c_tw[k];
   const int xb = (blockIdx.x % (N / XL)) * XL, y = blockIdx.x / (N / XL);
   const size_t base = (size_t)y * N + xb, zs = (size_t)N * N;
   // element e = threadIdx.x + r NT of the [z][16] tile: z = e / 16, x = e % 16
   const int ex = threadIdx.x % XL, ez = threadIdx.x / XL;
   constexpr int ZS = NT / XL;  // z rows per r step
#pragma unroll
   for (int c = 0; c < R; c += 8) {
      float2 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
         v[r] = g[base + (size_t)(ez + (c + r) * ZS) * zs + ex];
#pragma unroll
      for (int r = 0; r < 8; ++r)
         sm[fsig<T>(ez + (c + r) * ZS) * LD + ex] = v[r];
   }
   __syncthreads();
   const int line = threadIdx.x / T, t = threadIdx.x % T;
   float2 wt[N / T];
   fft_twiddles<N, T>(t, tw, wt);
   if (MODE != 1)
      fft_line<N, T, false>(sm + line, LD, t, tw, wt);
   if (MODE == 2) {
      __syncthreads();
#pragma unroll
      for (int c = 0; c < R; c += 8) {
         float f[8];
#pragma unroll
         for (int r = 0; r < 8; ++r)
            f[r] = infl[base + (size_t)(ez + (c + r) * ZS) * zs + ex];
#pragma unroll
         for (int r = 0; r < 8; ++r) {
            float2& v = sm[fsig<T>(ez + (c + r) * ZS) * LD + ex];
            v = make_float2(v.x * f[r], v.y * f[r]);
         }
      }
      __syncthreads();
   }
   if (MODE != 0)
      fft_line<N, T, true>(sm + line, LD, t, tw, wt);
   __syncthreads();
#pragma unroll
   for (int r = 0; r < R; ++r)
      g[base + (size_t)(ez + r * ZS) * zs + ex] = sm[fsig<T>(ez + r * ZS) * LD + ex];
}

// ---------------------------------------------------------------------------
// The same 2-D plane transform spread over a thread-block cluster of CL CTAs
// per z plane (N CL CTAs in all).  CTA r of the cluster stages rows
// [r R, r R + R) of the plane (R = N / CL), one contiguous R N-word slab,
// with one bulk asynchronous copy (cp.async.bulk, completion on an mbarrier
// with a bounded wait), transforms them along x, and after a cluster barrier
// gathers columns [r R, r R + R) of the whole plane from the R-row tiles of
// the CL CTAs through distributed shared memory; it transforms those along y
// and stores them.  The per-line arithmetic is fft_line's, in the same order
// as k_fft_plane, so the results are bit-identical to it.
template <int N, int CL>
struct PlaneCl {
   static constexpr int T = fft_threads_per_line<N>();
   static constexpr int R = N / CL;           // rows (and columns) per CTA
   static constexpr int NT = R * T;           // threads
   static constexpr int LDR = N + 2;          // row tile pitch (float2)
   static constexpr int LDC = R + 1;          // column tile pitch
   static constexpr int PER = R * N / NT;     // elements per thread in a tile copy
   static constexpr size_t STAGE = (size_t)R * N * 8;  // bytes of the staged slab
   static constexpr size_t SMEM = STAGE + sizeof(float2) * ((size_t)R * LDR + (size_t)N * LDC + 128) + 16;
};

template <int N, int CL, bool FROM_FX, bool INV>
__global__ void __launch_bounds__(PlaneCl<N, CL>::NT) k_fft_plane_cl(long long* __restrict__ qfx,
   float2* __restrict__ g, int packed, float inv, int* __restrict__ err)
{
   using C = PlaneCl<N, CL>;
   constexpr int T = C::T, R = C::R, NT = C::NT, LDR = C::LDR, LDC = C::LDC, PER = C::PER;
   extern __shared__ __align__(128) unsigned char smem_raw[];
   unsigned long long* stage = reinterpret_cast<unsigned long long*>(smem_raw);
   float2* rowt = reinterpret_cast<float2*>(smem_raw + C::STAGE);
   float2* colt = rowt + R * LDR;
   float2* tw = colt + N * LDC;
   unsigned long long* bar = reinterpret_cast<unsigned long long*>(tw + 128);
   unsigned rank;
   asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
   const int z = blockIdx.x / CL;
   const size_t base = (size_t)z * N * N + (size_t)rank * R * N;  // first word of this CTA's rows
   const unsigned bar_s = (unsigned)__cvta_generic_to_shared(bar);
   const unsigned stage_s = (unsigned)__cvta_generic_to_shared(stage);
   if (threadIdx.x == 0)
      mbar_init(bar_s, 1);
   __syncthreads();
   if (threadIdx.x == 0) {
      const void* src = FROM_FX ? static_cast<const void*>(qfx + base) : static_cast<const void*>(g + base);
      mbar_expect_tx(bar_s, (unsigned)C::STAGE);
      bulk_g2s(stage_s, src, (unsigned)C::STAGE, bar_s);
   }
   for (int k = threadIdx.x; k < 128; k += NT)
      tw[k] = c_tw[k];
   if (!mbar_wait_bounded(bar_s, 0)) {
      // the copy never completed: record it, wait once more for it, go on
      if (threadIdx.x == 0)
         atomicExch(err, 1);
      mbar_wait_bounded(bar_s, 0);
   }
   // staged slab -> row tile (element e: row e / N, column e % N)
#pragma unroll
   for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * NT;
      float2 v;
      if (FROM_FX)
         v = grid_word((long long)stage[e], packed, inv);
      else
         v = reinterpret_cast<const float2*>(stage)[e];
      rowt[(e / N) * LDR + fsig<T>(e % N)] = v;
   }
   if (FROM_FX) {
      // the fixed-point slab is cleared for the next spread
      long long* q = qfx + base;
#pragma unroll
      for (int k = 0; k < PER; ++k)
         q[threadIdx.x + k * NT] = 0;
   }
   __syncthreads();
   const int line = threadIdx.x / T, t = threadIdx.x % T;
   float2 wt[N / T];
   fft_twiddles<N, T>(t, tw, wt);
   fft_line<N, T, INV>(rowt + line * LDR, 1, t, tw, wt);  // row rank R + line, along x
   // every CTA's rows transformed before any column gather
   asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
   // columns [rank R, rank R + R) of all N rows, from the owners' row tiles;
   // all PER remote loads are issued before any store
   const unsigned rowt_s = (unsigned)__cvta_generic_to_shared(rowt);
   float2 v[PER];
#pragma unroll
   for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * NT;
      const int y = e / R, xl = e % R;
      const unsigned owner = (unsigned)(y / R);
      const unsigned local = rowt_s + (unsigned)(((y % R) * LDR + fsig<T>((int)rank * R + xl)) * sizeof(float2));
      unsigned remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(owner));
      // volatile keeps the loads after the cluster barrier; no memory clobber, so they pipeline
      asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[k].x), "=f"(v[k].y) : "r"(remote));
   }
#pragma unroll
   for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * NT;
      colt[fsig<T>(e / R) * LDC + e % R] = v[k];
   }
   __syncthreads();
   fft_line<N, T, INV>(colt + line, LDC, t, tw, wt);  // column rank R + line, along y
   __syncthreads();
   float2* out = g + (size_t)z * N * N + (size_t)rank * R;
#pragma unroll
   for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * NT;
      const int y = e / R, xl = e % R;
      out[(size_t)y * N + xl] = colt[fsig<T>(y) * LDC + xl];
   }
   // no CTA leaves while a peer may still read its row tile
   asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int N, int CL, bool FROM_FX, bool INV>
static cudaError_t launch_plane_cl(long long* qfx, float2* g, int packed, float inv, int* err, cudaStream_t st)
{
   using C = PlaneCl<N, CL>;
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(N * CL);
   cfg.blockDim = dim3(C::NT);
   cfg.dynamicSmemBytes = C::SMEM;
   cfg.stream = st;
   cudaLaunchAttribute at[1];
   at[0].id = cudaLaunchAttributeClusterDimension;
   at[0].val.clusterDim.x = CL;
   at[0].val.clusterDim.y = 1;
   at[0].val.clusterDim.z = 1;
   cfg.attrs = at;
   cfg.numAttrs = 1;
   return cudaLaunchKernelEx(&cfg, k_fft_plane_cl<N, CL, FROM_FX, INV>, qfx, g, packed, inv, err);
}

template <int N, int CL>
static int plane_cl_setup(Context* ctx)
{
   const int bytes = (int)PlaneCl<N, CL>::SMEM;
   T9_CUDA(cudaFuncSetAttribute(k_fft_plane_cl<N, CL, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      bytes));
   T9_CUDA(cudaFuncSetAttribute(k_fft_plane_cl<N, CL, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      bytes));
   return T9GB_OK;
}

template <int N>
static size_t fft_plane_smem()
{
   return sizeof(float2) * ((size_t)N * fft_plane_ld<N>() + 128);
}

// plane pass with clusters of P.fft_cl CTAs (0: one CTA per plane)
template <int N, bool FROM_FX, bool INV>
static void plane_pass(const PmeGrid& P, cudaStream_t st, int packed, float inv, bool pdl, int* range)
{
   constexpr int T = fft_threads_per_line<N>();
   if (P.fft_cl == 2)
      launch_plane_cl<N, 2, FROM_FX, INV>(P.qfx, P.qgrid, packed, inv, P.fft_err, st);
   else if (P.fft_cl == 4)
      launch_plane_cl<N, 4, FROM_FX, INV>(P.qfx, P.qgrid, packed, inv, P.fft_err, st);
   else if (P.fft_cl == 8)
      launch_plane_cl<N, 8, FROM_FX, INV>(P.qfx, P.qgrid, packed, inv, P.fft_err, st);
   else
      launch_k(pdl, k_fft_plane<N, FROM_FX, INV>, N, N * T, fft_plane_smem<N>(), st, P.qfx, P.qgrid, packed, inv,
         range);
}


template <int N>
static int fft_setup_kernels(Context* ctx)
{
   int rc = plane_cl_setup<N, 2>(ctx);
   if (rc == T9GB_OK)
      rc = plane_cl_setup<N, 4>(ctx);
   if (rc == T9GB_OK && N >= 64)
      rc = plane_cl_setup<N, 8>(ctx);
   T9_CHECK(rc);
   const int bytes = (int)fft_plane_smem<N>();
   void (*fwd)(long long*, float2*, int, float, int*) = k_fft_plane<N, true, false>;
   void (*inv)(long long*, float2*, int, float, int*) = k_fft_plane<N, false, true>;
   T9_CUDA(cudaFuncSetAttribute(fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
   T9_CUDA(cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
   return T9GB_OK;
}

// forward planes; vir: the z pass stops after the forward transform
template <int N>
static void fft_own_forward(const PmeGrid& P, cudaStream_t st, bool split, bool pdl, int* range)
{
   constexpr int T = fft_threads_per_line<N>();
   plane_pass<N, true, false>(P, st, P.packed ? 1 : 0, 1.0f / (float)(1 << P.pack_shift), pdl, range);
   if (split)
      launch_k(pdl, k_fft_zline<N, 0>, N * N / 16, 16 * T, 0, st, P.infl, P.qgrid);
   else
      launch_k(pdl, k_fft_zline<N, 2>, N * N / 16, 16 * T, 0, st, P.infl, P.qgrid);
}

template <int N>
static void fft_own_inverse(const PmeGrid& P, cudaStream_t st, bool split, bool pdl)
{
   constexpr int T = fft_threads_per_line<N>();
   if (split)
      launch_k(pdl, k_fft_zline<N, 1>, N * N / 16, 16 * T, 0, st, P.infl, P.qgrid);
   plane_pass<N, false, true>(P, st, 0, 0.f, pdl, nullptr);
}

// ---------------------------------------------------------------------------
// Small cubic grids: the conversion from fixed point, the 3-D FFT, the
// convolution and the inverse FFT as one kernel, on one cluster of SG_CL CTAs
// that keeps the grid in its shared memory.  CTA r has planes
// [r N / SG_CL, ...) for the x and y passes; for the z passes it has columns
// [r N^2 / SG_CL, ...), which it reads from its peers' planes and writes back
// through distributed shared memory.  An edge is RA x RB, each 2 to 8, and a
// pass two Stockham steps between two buffers: for the factor R after the
// product S of the factors before it, butterfly j takes the elements
// j + q N / R and writes (j / S) S R + j % S + q S.  The inverse transform is
// the forward one with real and imaginary parts exchanged before and after.
//
// What bounds it: a chain of twelve steps with a barrier each (about 250
// cycles at 24^3, where a step moves 14 KB through a CTA's shared memory in
// 110 of them; at 40^3 it moves 64 KB and the shared memory bounds it), two
// cluster barriers and one trip to global memory each way.  It takes the
// place of eight launches of a few microseconds (cuFFT's six, conversion,
// convolution): a solve of 648 atoms from alpha E on 16 / 18 / 20 / 24 / 30 /
// 36 / 40 points an edge takes 247 / 273 / 254 / 262 / 272 / 299 / 337 us instead
// of 350 / 357 / 362 / 356 / 375 / 360 / 371, and on 32 points 268 instead of the
// 282 of the plane kernels.  8 CTAs take 7 / 30 / 38 us more than 16 at 24 / 30 /
// 40, 256 threads 2 / 15 / 33 more than 512.  Edges are known at compile time:
// the same steps with factors and strides from a table took 17.7 us a
// transform at 24^3 instead of 7.3.
constexpr int SG_CL = 16;       // CTAs, the largest cluster
constexpr int SG_THREADS = 512;

template <int R>
__device__ __forceinline__ void dft_small(float2* v)
{
   if constexpr (R == 2) {
      const float2 a = v[0], b = v[1];
      v[0] = make_float2(a.x + b.x, a.y + b.y);
      v[1] = make_float2(a.x - b.x, a.y - b.y);
   } else if constexpr (R == 3) {
      const float s3 = 0.866025403784438647f;
      const float2 t = make_float2(v[1].x + v[2].x, v[1].y + v[2].y);
      const float2 d = make_float2(s3 * (v[1].x - v[2].x), s3 * (v[1].y - v[2].y));
      const float2 m = make_float2(v[0].x - 0.5f * t.x, v[0].y - 0.5f * t.y);
      v[0] = make_float2(v[0].x + t.x, v[0].y + t.y);
      v[1] = make_float2(m.x + d.y, m.y - d.x);
      v[2] = make_float2(m.x - d.y, m.y + d.x);
   } else if constexpr (R == 4) {
      const float2 a = make_float2(v[0].x + v[2].x, v[0].y + v[2].y), b = make_float2(v[0].x - v[2].x, v[0].y - v[2].y);
      const float2 c = make_float2(v[1].x + v[3].x, v[1].y + v[3].y), d = make_float2(v[1].x - v[3].x, v[1].y - v[3].y);
      v[0] = make_float2(a.x + c.x, a.y + c.y);
      v[1] = make_float2(b.x + d.y, b.y - d.x);
      v[2] = make_float2(a.x - c.x, a.y - c.y);
      v[3] = make_float2(b.x - d.y, b.y + d.x);
   } else if constexpr (R == 5) {
      // cos and sin of 2 pi / 5 and 4 pi / 5
      const float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f;
      const float s1 = 0.951056516295153572f, s2 = 0.587785252292473129f;
      const float2 a = make_float2(v[1].x + v[4].x, v[1].y + v[4].y), b = make_float2(v[1].x - v[4].x, v[1].y - v[4].y);
      const float2 c = make_float2(v[2].x + v[3].x, v[2].y + v[3].y), d = make_float2(v[2].x - v[3].x, v[2].y - v[3].y);
      const float2 p = make_float2(v[0].x + c1 * a.x + c2 * c.x, v[0].y + c1 * a.y + c2 * c.y);
      const float2 q = make_float2(v[0].x + c2 * a.x + c1 * c.x, v[0].y + c2 * a.y + c1 * c.y);
      const float2 e = make_float2(s1 * b.x + s2 * d.x, s1 * b.y + s2 * d.y);
      const float2 f = make_float2(s2 * b.x - s1 * d.x, s2 * b.y - s1 * d.y);
      v[0] = make_float2(v[0].x + a.x + c.x, v[0].y + a.y + c.y);
      v[1] = make_float2(p.x + e.y, p.y - e.x);
      v[4] = make_float2(p.x - e.y, p.y + e.x);
      v[2] = make_float2(q.x + f.y, q.y - f.x);
      v[3] = make_float2(q.x - f.y, q.y + f.x);
   } else {
      // R = 6, 8: the halves of even and odd index
      constexpr int H = R / 2;
      float2 e[H], o[H];
#pragma unroll
      for (int k = 0; k < H; ++k) {
         e[k] = v[2 * k];
         o[k] = v[2 * k + 1];
      }
      dft_small<H>(e);
      dft_small<H>(o);
#pragma unroll
      for (int k = 0; k < H; ++k) {
         constexpr float h = 0.5f, s3 = 0.866025403784438647f, r2 = 0.707106781186547524f;
         const float2 w = H == 3 ? (k == 0 ? make_float2(1.f, 0.f) : (k == 1 ? make_float2(h, -s3) : make_float2(-h, -s3)))
                                 : (k == 0 ? make_float2(1.f, 0.f)
                                           : (k == 1 ? make_float2(r2, -r2)
                                                     : (k == 2 ? make_float2(0.f, -1.f) : make_float2(-r2, -r2))));
         const float2 t = k == 0 ? o[0] : (H == 4 && k == 2 ? make_float2(o[2].y, -o[2].x) : cmulf(w, o[k]));
         v[k] = make_float2(e[k].x + t.x, e[k].y + t.y);
         v[k + H] = make_float2(e[k].x - t.x, e[k].y - t.y);
      }
   }
}

template <int N>
struct SmallGrid {
   static constexpr int P = N | 1;  // row pitch: odd, so that threads on consecutive rows meet different banks
   static constexpr int NZ = (N + SG_CL - 1) / SG_CL;       // the most planes of a CTA
   static constexpr int NC = (N * N + SG_CL - 1) / SG_CL;   // the most columns
   static constexpr int BUF = NZ * N * P > NC * N ? NZ * N * P : NC * N;
   static constexpr size_t SMEM = sizeof(float2) * (2 * BUF + NC * N + N);
   __device__ __forceinline__ static int z_owner(int z) { return ((z + 1) * SG_CL - 1) / N; }
   __device__ __forceinline__ static int z_first(int r) { return r * N / SG_CL; }
};

// one Stockham step of the first `lines` of at most LM lines; load(l, i) and
// store(l, i, k, v) take element i of line l (k: the thread's count of stores)
template <int N, int R, int S, int LM, class Load, class Store>
__device__ __forceinline__ void sg_step(int lines, const float2* tw, Load load, Store store)
{
   constexpr int NJ = N / R, TASKS = (LM * NJ + SG_THREADS - 1) / SG_THREADS;
#pragma unroll
   for (int it = 0; it < TASKS; ++it) {
      const int t = threadIdx.x + it * SG_THREADS, j = t / LM, l = t % LM;
      if (j >= NJ || l >= lines)
         continue;
      const int jl = j % S, to = j / S * S * R + jl;
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q)
         v[q] = load(l, j + q * NJ);
      if (S > 1)
#pragma unroll
         for (int q = 1; q < R; ++q)
            v[q] = cmulf(v[q], tw[q * jl * (N / (S * R))]);
      dft_small<R>(v);
#pragma unroll
      for (int q = 0; q < R; ++q)
         store(l, to + q * S, it * R + q, v[q]);
   }
}

template <int N, int RA, int RB>
__global__ void __launch_bounds__(SG_THREADS) k_fft_small(long long* __restrict__ qfx, float2* __restrict__ g,
   const float* __restrict__ infl, const float2* __restrict__ twg, int packed, float inv, int* __restrict__ range)
{
   using G = SmallGrid<N>;
   constexpr int P = G::P, NC = G::NC, LX = G::NZ * N;
   constexpr int PER = (G::NZ * N * N + SG_THREADS - 1) / SG_THREADS;       // grid points a thread
   constexpr int CT = (NC * RA + SG_THREADS - 1) / SG_THREADS;              // z tasks of the second step
   extern __shared__ __align__(16) float2 sgm[];
   float2* const b0 = sgm;  // planes, read and written by the peers
   float2* const b1 = b0 + G::BUF;
   float2* const b2 = b1 + G::BUF;
   float2* const tw = b2 + NC * N;
   unsigned rank;
   asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
   const int z0 = G::z_first((int)rank), nz = G::z_first((int)rank + 1) - z0;
   const int c0 = (int)rank * N * N / SG_CL, nc = ((int)rank + 1) * N * N / SG_CL - c0;
   const int tid = threadIdx.x;
   if (tid < N)
      tw[tid] = twg[tid];
   // the influence function where this thread's second z step will need it
   float fn[CT * RB];
#pragma unroll
   for (int it = 0; it < CT; ++it) {
      const int t = tid + it * SG_THREADS, j = t / NC, l = t % NC;
#pragma unroll
      for (int q = 0; q < RB; ++q)
         fn[it * RB + q] = j < RA && l < nc ? infl[(size_t)(j + q * RA) * N * N + c0 + l] : 0.f;
   }
   pdl_wait();
   pdl_trigger();
   bool big = false;
   {
      long long* q = qfx + (size_t)z0 * N * N;
      long long w[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k)
         w[k] = tid + k * SG_THREADS < nz * N * N ? q[tid + k * SG_THREADS] : 0;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
         const int e = tid + k * SG_THREADS;
         if (e >= nz * N * N)
            continue;
         q[e] = 0;
         big |= grid_word_big(w[k], packed);
         b0[e / N * P + e % N] = grid_word(w[k], packed, inv);
      }
   }
   if (big)
      atomicOr(range, 1);
   __syncthreads();
   // plane passes from b0 over b1 back to b0; element i of row l, of column
   // (plane l / N, x l % N)
   auto px = [](int l, int i) { return l * P + i; };
   auto py = [](int l, int i) { return l / N * (N * P) + i * P + l % N; };
   auto plane = [&](auto at) {
      sg_step<N, RA, 1, LX>(nz * N, tw, [&](int l, int i) { return b0[at(l, i)]; },
         [&](int l, int i, int, float2 v) { b1[at(l, i)] = v; });
      __syncthreads();
      sg_step<N, RB, RA, LX>(nz * N, tw, [&](int l, int i) { return b1[at(l, i)]; },
         [&](int l, int i, int, float2 v) { b0[at(l, i)] = v; });
   };
   plane(px);
   __syncthreads();
   plane(py);
   asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
   // point (z, column c0 + l) in its owner's b0
   const unsigned b0_s = (unsigned)__cvta_generic_to_shared(b0);
   auto peer = [&](int l, int z) {
      const int own = G::z_owner(z), c = c0 + l;
      const unsigned at = b0_s + 8u * (unsigned)(((z - G::z_first(own)) * N + c / N) * P + c % N);
      unsigned r;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"((unsigned)own));
      return r;
   };
   sg_step<N, RA, 1, NC>(nc, tw,
      [&](int l, int z) {
         float2 v;
         // volatile keeps the loads after the barrier; no memory clobber, so they pipeline
         asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(peer(l, z)));
         return v;
      },
      [&](int l, int z, int, float2 v) { b1[z * NC + l] = v; });
   __syncthreads();
   // the convolution, and the exchange of real and imaginary parts
   sg_step<N, RB, RA, NC>(nc, tw, [&](int l, int z) { return b1[z * NC + l]; },
      [&](int l, int z, int k, float2 v) { b2[z * NC + l] = make_float2(v.y * fn[k], v.x * fn[k]); });
   __syncthreads();
   sg_step<N, RA, 1, NC>(nc, tw, [&](int l, int z) { return b2[z * NC + l]; },
      [&](int l, int z, int, float2 v) { b1[z * NC + l] = v; });
   __syncthreads();
   // a column belongs to one CTA: no peer still reads what is written here
   sg_step<N, RB, RA, NC>(nc, tw, [&](int l, int z) { return b1[z * NC + l]; },
      [&](int l, int z, int, float2 v) {
         asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(peer(l, z)), "f"(v.x), "f"(v.y) : "memory");
      });
   asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
   plane(py);
   __syncthreads();
   plane(px);
   __syncthreads();
#pragma unroll
   for (int k = 0; k < PER; ++k) {
      const int e = tid + k * SG_THREADS;
      if (e < nz * N * N) {
         const float2 v = b0[e / N * P + e % N];
         g[(size_t)z0 * N * N + e] = make_float2(v.y, v.x);
      }
   }
}

using SmallFft = void (*)(long long*, float2*, const float*, const float2*, int, float, int*);

// The kernel of an edge and its shared memory; null: not a small grid.  Even
// products of two factors, from 16 (the least edge of a box with a 7 A
// cutoff) to 40: at 48 the gain is down to 8 % (384 for 419 us) and the
// trajectories' sensitivity to rounding, which grows with the box, moves the
// velocities of a restart by 1.6e-5 between the two transforms (1.2e-5 at
// 40), so larger boxes keep the transform they had.
static SmallFft small_fft_kernel(int n, size_t* smem)
{
   switch (n) {
   case 16: *smem = SmallGrid<16>::SMEM; return k_fft_small<16, 4, 4>;
   case 18: *smem = SmallGrid<18>::SMEM; return k_fft_small<18, 3, 6>;
   case 20: *smem = SmallGrid<20>::SMEM; return k_fft_small<20, 4, 5>;
   case 24: *smem = SmallGrid<24>::SMEM; return k_fft_small<24, 4, 6>;
   case 30: *smem = SmallGrid<30>::SMEM; return k_fft_small<30, 5, 6>;
   case 32: *smem = SmallGrid<32>::SMEM; return k_fft_small<32, 4, 8>;
   case 36: *smem = SmallGrid<36>::SMEM; return k_fft_small<36, 6, 6>;
   case 40: *smem = SmallGrid<40>::SMEM; return k_fft_small<40, 5, 8>;
   }
   return nullptr;
}

// the launch as one cluster; at: room for its attributes
static cudaLaunchConfig_t small_fft_config(size_t smem, cudaLaunchAttribute* at)
{
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(SG_CL);
   cfg.blockDim = dim3(SG_THREADS);
   cfg.dynamicSmemBytes = smem;
   at[0].id = cudaLaunchAttributeClusterDimension;
   at[0].val.clusterDim.x = SG_CL;
   at[0].val.clusterDim.y = 1;
   at[0].val.clusterDim.z = 1;
   cfg.attrs = at;
   cfg.numAttrs = 1;
   return cfg;
}

static int launch_small_fft(Context* ctx, int* range)
{
   PmeGrid& P = ctx->pme;
   size_t smem = 0;
   const SmallFft k = small_fft_kernel(P.n1, &smem);
   cudaLaunchAttribute at[2];
   cudaLaunchConfig_t cfg = small_fft_config(smem, at);
   cfg.stream = ctx->stream;
   at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   at[1].val.programmaticStreamSerializationAllowed = 1;
   cfg.numAttrs = use_pdl(ctx) ? 2 : 1;
   T9_CUDA(cudaLaunchKernelEx(&cfg, k, P.qfx, P.qgrid, (const float*)P.infl, (const float2*)P.small_tw,
      P.packed ? 1 : 0, 1.0f / (float)(1 << P.pack_shift), range));
   return T9GB_OK;
}

static int small_fft_setup(Context* ctx)
{
   PmeGrid& P = ctx->pme;
   size_t smem = 0;
   const SmallFft k = P.n1 == P.n2 && P.n2 == P.n3 ? small_fft_kernel(P.n1, &smem) : nullptr;
   if (!k)
      return T9GB_OK;
   std::vector<float2> tw(P.n1);
   for (int i = 0; i < P.n1; ++i) {
      const double x = 2 * 3.14159265358979323846 * i / P.n1;
      tw[i] = make_float2((float)std::cos(x), (float)-std::sin(x));
   }
   T9_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
   T9_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
   cudaLaunchAttribute at;
   cudaLaunchConfig_t cfg = small_fft_config(smem, &at);
   int fit = 0;
   if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();  // a device whose free SMs hold no such cluster keeps cuFFT or the planes
      return T9GB_OK;
   }
   T9_CUDA(cudaMalloc(&P.small_tw, sizeof(float2) * tw.size()));
   T9_CUDA(cudaMemcpy(P.small_tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice));
   return T9GB_OK;
}

// ---------------------------------------------------------------------------
// k-space part of the reciprocal virial (the strain derivative of the
// influence function), read-only on the forward-transformed grid:
//   W_ab += sum_m w(m) G(m) [-delta_ab + 2 h_a h_b (1 + pi^2 h^2 / a^2) / h^2]
// MODE 1 (permanent grid): w = wE |F(m)|^2, and the grid is kept in qstash
// when stash != null.  MODE 2 (d real, p imaginary): with
// Q_d = (F(m) + F*(-m)) / 2, Q_p = (F(m) - F*(-m)) / 2i and the kept
// permanent Q_M, w = wP Re[Q_M (Q_d + Q_p)* + Q_d Q_p*].  The reference's
// counterpart is pmeConv_cu1<Do_V> (src/cu/pme.cu:908-1031).  Six sums in a
// fixed order; the last block writes them to out[0..6) (xx yy zz xy xz yz).
template <int MODE>
__global__ void k_conv_virial(int n1, int n2, int n3, float L1, float L2, float L3, float pterm,
   const float* __restrict__ infl, const float2* __restrict__ g, float2* __restrict__ stash, float wE, float wP,
   double* __restrict__ red, double* __restrict__ out, int* __restrict__ state)
{
   __shared__ double sh[64];
   float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // FP32 per thread and warp, FP64 above
   const size_t ng = (size_t)n1 * n2 * n3;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ng; i += (size_t)gridDim.x * blockDim.x) {
      const int k1 = (int)(i % n1), k2 = (int)((i / n1) % n2), k3 = (int)(i / ((size_t)n1 * n2));
      const float2 F = g[i];
      float2 QM = make_float2(0.f, 0.f);
      if (MODE == 1 && stash)
         stash[i] = F;
      if (MODE == 2)
         QM = stash[i];
      if (i == 0)
         continue;
      const int r1 = (k1 < (n1 + 1) / 2) ? k1 : k1 - n1;
      const int r2 = (k2 < (n2 + 1) / 2) ? k2 : k2 - n2;
      const int r3 = (k3 < (n3 + 1) / 2) ? k3 : k3 - n3;
      const float h[3] = {r1 / L1, r2 / L2, r3 / L3};
      const float hsq = h[0] * h[0] + h[1] * h[1] + h[2] * h[2];
      // per-point terms in FP32; the block and grid sums in FP64
      float w;
      if (MODE == 1) {
         w = wE * (F.x * F.x + F.y * F.y);
      } else {
         const int m1 = k1 == 0 ? 0 : n1 - k1, m2 = k2 == 0 ? 0 : n2 - k2, m3 = k3 == 0 ? 0 : n3 - k3;
         const float2 Fm = g[((size_t)m3 * n2 + m2) * n1 + m1];
         // Q_d = (F + conj(Fm)) / 2, Q_p = (F - conj(Fm)) / (2i)
         const float dx = 0.5f * (F.x + Fm.x), dy = 0.5f * (F.y - Fm.y);
         const float px = 0.5f * (F.y + Fm.y), py = -0.5f * (F.x - Fm.x);
         const float ux = dx + px, uy = dy + py;
         w = wP * ((QM.x * ux + QM.y * uy) + (dx * px + dy * py));
      }
      w *= infl[i];
      const float wf = w * (2.f * (1.f + pterm * hsq) / hsq);
      v[0] += wf * h[0] * h[0] - w;
      v[1] += wf * h[1] * h[1] - w;
      v[2] += wf * h[2] * h[2] - w;
      v[3] += wf * h[0] * h[1];
      v[4] += wf * h[0] * h[2];
      v[5] += wf * h[1] * h[2];
   }
   store_partials_f<6>(red, 0, v, sh);
   if (!last_block(state + ST_TICKET0))
      return;
   double t[4];
   sum_slots(red, 0, 4, gridDim.x, sh, t);
   double t2[4];
   sum_slots(red, 4, 2, gridDim.x, sh, t2);
   if (threadIdx.x == 0) {
      out[0] = t[0];
      out[1] = t[1];
      out[2] = t[2];
      out[3] = t[3];
      out[4] = t2[0];
      out[5] = t2[1];
   }
}

// ---------------------------------------------------------------------------
// Force gathers: the 20 fractional derivatives of the reciprocal potential
// (level-4 weights; the reference's fphi order: 0, x, y, z, xx, yy, zz, xy,
// xz, yz, xxx, yyy, zzz, xxy, xxz, xyy, yyz, xzz, yzz, xyz), made Cartesian
// (orthogonal box: one factor nfft/L per derivative) and contracted on the
// spot.  Replaces fphiMpole/fphiUind (src/cu/pme.cu:383-906) followed by the
// force/torque parts of empoleEwaldRecipGeneric_cu (src/cu/hippo/empole.cu)
// and epolarEwaldRecipSelf_cu1 (src/cu/epolarrecip.cu:414-511).

__device__ __forceinline__ void fphi20(const float* t, const float* u, const float* v, float* phi)
{
   phi[0] = t[0] * u[0] * v[0];
   phi[1] = t[1] * u[0] * v[0];
   phi[2] = t[0] * u[1] * v[0];
   phi[3] = t[0] * u[0] * v[1];
   phi[4] = t[2] * u[0] * v[0];
   phi[5] = t[0] * u[2] * v[0];
   phi[6] = t[0] * u[0] * v[2];
   phi[7] = t[1] * u[1] * v[0];
   phi[8] = t[1] * u[0] * v[1];
   phi[9] = t[0] * u[1] * v[1];
   phi[10] = t[3] * u[0] * v[0];
   phi[11] = t[0] * u[3] * v[0];
   phi[12] = t[0] * u[0] * v[3];
   phi[13] = t[2] * u[1] * v[0];
   phi[14] = t[2] * u[0] * v[1];
   phi[15] = t[1] * u[2] * v[0];
   phi[16] = t[0] * u[2] * v[1];
   phi[17] = t[1] * u[0] * v[2];
   phi[18] = t[0] * u[1] * v[2];
   phi[19] = t[1] * u[1] * v[1];
}

// fractional -> Cartesian for the 20 derivatives
__device__ __forceinline__ void to_cart20(const GridParams& G, float* c)
{
   const float a = G.a1, b = G.a2, d = G.a3;
   c[1] *= a;
   c[2] *= b;
   c[3] *= d;
   c[4] *= a * a;
   c[5] *= b * b;
   c[6] *= d * d;
   c[7] *= a * b;
   c[8] *= a * d;
   c[9] *= b * d;
   c[10] *= a * a * a;
   c[11] *= b * b * b;
   c[12] *= d * d * d;
   c[13] *= a * a * b;
   c[14] *= a * a * d;
   c[15] *= a * b * b;
   c[16] *= b * b * d;
   c[17] *= a * d * d;
   c[18] *= b * d * d;
   c[19] *= a * b * d;
}

__device__ __forceinline__ int ix2(int a, int b)
{
   return a == b ? 4 + a : (a + b == 1 ? 7 : (a + b == 2 ? 8 : 9));
}

__device__ __forceinline__ int ix3(int a, int b, int c)
{
   int n[3] = {0, 0, 0};
   n[a]++;
   n[b]++;
   n[c]++;
   if (n[0] == 3)
      return 10;
   if (n[1] == 3)
      return 11;
   if (n[2] == 3)
      return 12;
   if (n[0] == 2)
      return n[1] ? 13 : 14;
   if (n[1] == 2)
      return n[0] ? 15 : 16;
   if (n[2] == 2)
      return n[0] ? 17 : 18;
   return 19;
}

// -(q phi_a + d_b phi_ab + Theta_bc phi_abc) for a multipole row m (12 floats)
__device__ __forceinline__ void mpole_force(const float* m, const float* c, float* F)
{
   const float Q[3][3] = {{m[4], m[7], m[8]}, {m[7], m[5], m[9]}, {m[8], m[9], m[6]}};
#pragma unroll
   for (int a = 0; a < 3; ++a) {
      float v = m[0] * c[1 + a];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
         v += m[1 + b] * c[ix2(a, b)];
#pragma unroll
         for (int cc = 0; cc < 3; ++cc)
            v += Q[b][cc] * c[ix3(a, b, cc)];
      }
      F[a] = -v;
   }
}

// The 20 sums of one atom over its 125 points (IMAG: of both parts), value k
// left in out[k] (out[20 + k] the imaginary part's), shared memory.  The points
// are loaded and exchanged as in gather_atom; lane (jy, kz) then sums its row
// with the four x levels, forms its 20 products and the halving tree adds the
// rows in the order of an xor tree (23 shuffles where 20 trees take 100).
template <bool IMAG>
__device__ __forceinline__ void force_sums(int s, int lane, const GridParams& G, const Sites& S,
   const float2* __restrict__ g, float2* xch, float* out)
{
   const int4 o = S.org[s];
   const float* lo = S.lo + (size_t)SPL_ROW * s;
   const float* hi = S.hi + (size_t)SPL_ROW * s;
   const int q5 = lane % 5, d5 = lane / 5;  // (ix, jy) loading, (jy, kz) summing
   float* xr = reinterpret_cast<float*>(xch);
   if (lane < 25) {
      const unsigned plane = plane_bytes(G);
      const char* col = reinterpret_cast<const char*>(g) + column_bytes(G, o, q5, d5);
      float2 q[5];
#pragma unroll
      for (int kz = 0; kz < 5; ++kz) {
         int zb = o.z + kz;
         zb -= (zb >= G.n3 ? G.n3 : 0);
         const float2* p = reinterpret_cast<const float2*>(col + (size_t)(unsigned)zb * plane);
         if (IMAG)
            q[kz] = *p;
         else
            q[kz].x = p->x;
      }
#pragma unroll
      for (int kz = 0; kz < 5; ++kz)
         if (IMAG)
            xch[25 * kz + lane] = q[kz];
         else
            xr[25 * kz + lane] = q[kz].x;
   }
   __syncwarp();
   float phi[20], psi[20];
#pragma unroll
   for (int c = 0; c < 20; ++c)
      phi[c] = psi[c] = 0.f;
   if (lane < 25) {
      float t[4] = {0.f, 0.f, 0.f, 0.f}, w[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ix = 0; ix < 5; ++ix) {
         const float2 a = spl(lo, 0, ix), b = spl(hi, 0, ix);
         float2 qv;
         if (IMAG)
            qv = xch[5 * lane + ix];
         else
            qv.x = xr[5 * lane + ix];
         t[0] += qv.x * a.x;
         t[1] += qv.x * a.y;
         t[2] += qv.x * b.x;
         t[3] += qv.x * b.y;
         if (IMAG) {
            w[0] += qv.y * a.x;
            w[1] += qv.y * a.y;
            w[2] += qv.y * b.x;
            w[3] += qv.y * b.y;
         }
      }
      const float2 ua = spl(lo, 1, q5), ub = spl(hi, 1, q5), va = spl(lo, 2, d5), vb = spl(hi, 2, d5);
      const float u[4] = {ua.x, ua.y, ub.x, ub.y}, v[4] = {va.x, va.y, vb.x, vb.y};
      fphi20(t, u, v, phi);
      if (IMAG)
         fphi20(w, u, v, psi);
   }
   const float a = warp_sums<20>(phi, lane);
   const int c = sum_slot<20>(lane);
   if (c >= 0)
      out[c] = a;
   if (IMAG) {
      const float b = warp_sums<20>(psi, lane);
      if (c >= 0)
         out[20 + c] = b;
   }
   __syncwarp();
}

// Each warp sums FA consecutive atoms, then its first FA lanes finish one atom
// each (one lane finishing each atom as it is summed takes 300 to 400 warp
// instructions an atom).
constexpr int FORCE_WARPS = 8;

// permanent grid: multipole forces, torque field and energies (MPOLE), the
// polarization force on the dipoles in the permanent field gradient and the
// Ewald self torque (POLAR)
// wout (may be null): the fractional-transform part of the virial per slot,
// [9][npad]; the dipole-grid gather adds to the same rows
template <bool MPOLE, bool POLAR, int FA>
__global__ void __launch_bounds__(32 * FORCE_WARPS) k_gather_force_perm(int n, int npad, GridParams G, float f,
   float aewald, Sites S, const float2* __restrict__ g, const float* __restrict__ rp,
   const float* __restrict__ u8, float* __restrict__ fout, float* __restrict__ tout, double* __restrict__ e_atom,
   double* __restrict__ e_self, float* __restrict__ wout)
{
   __shared__ float2 xch[FORCE_WARPS][125];
   __shared__ float sums[FORCE_WARPS][FA][21];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const int s0 = (blockIdx.x * FORCE_WARPS + w) * FA;
   for (int a = 0; a < FA && s0 + a < n; ++a)
      force_sums<false>(s0 + a, lane, G, S, g, xch[w], sums[w][a]);
   const int s = s0 + lane;
   if (lane >= FA || s >= n)
      return;
   float phi[20];
#pragma unroll
   for (int c = 0; c < 20; ++c)
      phi[c] = sums[w][lane][c];
   to_cart20(G, phi);
   const float* m = rp + 12 * s;
   float F[3] = {0.f, 0.f, 0.f}, T[10];
#pragma unroll
   for (int c = 0; c < 10; ++c)
      T[c] = 0.f;
   if (MPOLE) {
      mpole_force(m, phi, F);
      #pragma unroll
      for (int c = 0; c < 3; ++c)
         F[c] *= f;
      #pragma unroll
      for (int c = 0; c < 10; ++c)
         T[c] = f * phi[c];
      // per-atom energies in FP32 (this GPU's FP64 pipe issues a warp
      // instruction in tens of cycles even for one lane); the totals are
      // FP64 sums of these
      if (e_atom) {
         float e = m[0] * phi[0] + m[1] * phi[1] + m[2] * phi[2] + m[3] * phi[3];
         e += m[4] * phi[4] + m[5] * phi[5] + m[6] * phi[6];
         e += 2.f * (m[7] * phi[7] + m[8] * phi[8] + m[9] * phi[9]);
         e_atom[s] = (double)(0.5f * f * e);
      }
      if (e_self) {
         const float a2 = 2.f * aewald * aewald;
         const float fterm = -f * aewald * 0.56418958354775628f;  // 1/sqrt(pi)
         const float cii = m[0] * m[0];
         const float dii = m[1] * m[1] + m[2] * m[2] + m[3] * m[3];
         const float qii = 2.f * (m[7] * m[7] + m[8] * m[8] + m[9] * m[9]) + m[4] * m[4] + m[5] * m[5] + m[6] * m[6];
         e_self[s] = (double)(fterm * (cii + a2 * (dii * (1.f / 3.f) + 0.4f * a2 * qii)));
      }
   }
   float us[3] = {0.f, 0.f, 0.f};
   if (POLAR) {
      const float* u = u8 + 8 * s;
      us[0] = u[0] + u[3];
      us[1] = u[1] + u[4];
      us[2] = u[2] + u[5];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
         float v = 0.f;
#pragma unroll
         for (int b = 0; b < 3; ++b)
            v += us[b] * phi[ix2(a, b)];
         F[a] -= 0.5f * f * v;
         T[1 + a] -= 0.5f * f * G.selfterm * us[a];
      }
   }
   #pragma unroll
   for (int c = 0; c < 3; ++c)
      fout[3 * s + c] = F[c];
   #pragma unroll
   for (int c = 0; c < 10; ++c)
      tout[10 * s + c] = T[c];
   if (wout) {
      // -f [phi_a d_b + 2 (phi2 Theta)_ab] (MPOLE), -f/2 phi_a u_b (POLAR)
      const float Q[3][3] = {{m[4], m[7], m[8]}, {m[7], m[5], m[9]}, {m[8], m[9], m[6]}};
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
         for (int b = 0; b < 3; ++b) {
            float w = 0.f;
            if (MPOLE) {
               float pq = 0.f;
#pragma unroll
               for (int c = 0; c < 3; ++c)
                  pq += phi[ix2(a, c)] * Q[c][b];
               w -= f * (phi[1 + a] * m[1 + b] + 2.f * pq);
            }
            if (POLAR)
               w -= 0.5f * f * phi[1 + a] * us[b];
            wout[(3 * a + b) * npad + s] = w;
         }
   }
}

// induced-dipole grid (d real, p imaginary): force on the multipoles in the
// dipoles' potential, the mutual dipole force and the torque field
template <int FA>
__global__ void __launch_bounds__(32 * FORCE_WARPS) k_gather_force_uind(int n, int npad, GridParams G, float f,
   Sites S, const float2* __restrict__ g, const float* __restrict__ rp,
   const float* __restrict__ u8, float* __restrict__ fout, float* __restrict__ tout, float* __restrict__ wout)
{
   __shared__ float2 xch[FORCE_WARPS][125];
   __shared__ float sums[FORCE_WARPS][FA][41];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const int s0 = (blockIdx.x * FORCE_WARPS + w) * FA;
   for (int a = 0; a < FA && s0 + a < n; ++a)
      force_sums<true>(s0 + a, lane, G, S, g, xch[w], sums[w][a]);
   const int s = s0 + lane;
   if (lane >= FA || s >= n)
      return;
   float pd[20], pp[20];
#pragma unroll
   for (int c = 0; c < 20; ++c) {
      pd[c] = sums[w][lane][c];
      pp[c] = sums[w][lane][20 + c];
   }
   to_cart20(G, pd);
   to_cart20(G, pp);
   float ps[20];
   #pragma unroll
   for (int c = 0; c < 20; ++c)
      ps[c] = pd[c] + pp[c];
   const float* m = rp + 12 * s;
   const float* u = u8 + 8 * s;
   float F[3];
   mpole_force(m, ps, F);
#pragma unroll
   for (int a = 0; a < 3; ++a) {
      float v = 0.f;
#pragma unroll
      for (int b = 0; b < 3; ++b)
         v += u[b] * pp[ix2(a, b)] + u[3 + b] * pd[ix2(a, b)];
      fout[3 * s + a] = 0.5f * f * (F[a] - v);
   }
   #pragma unroll
   for (int c = 0; c < 10; ++c)
      tout[10 * s + c] = 0.5f * f * ps[c];
   if (wout) {
      // -f/2 [psi_a d_b + 2 (psi2 Theta)_ab + psi^p_a u_d,b + psi^d_a u_p,b]
      const float Q[3][3] = {{m[4], m[7], m[8]}, {m[7], m[5], m[9]}, {m[8], m[9], m[6]}};
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
         for (int b = 0; b < 3; ++b) {
            float pq = 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c)
               pq += ps[ix2(a, c)] * Q[c][b];
            const float w = ps[1 + a] * m[1 + b] + 2.f * pq + pp[1 + a] * u[b] + pd[1 + a] * u[3 + b];
            wout[(3 * a + b) * npad + s] -= 0.5f * f * w;
         }
   }
}

// ---------------------------------------------------------------------------

int pme_setup(Context* ctx)
{
   const t9gb_config& c = ctx->cfg;
   PmeGrid& P = ctx->pme;
   if (!c.use_ewald)
      return T9GB_OK;
   P.n1 = c.nfft[0];
   P.n2 = c.nfft[1];
   P.n3 = c.nfft[2];
   const size_t ng = (size_t)P.n1 * P.n2 * P.n3;
   T9_CUDA(cudaMalloc(&P.qgrid, sizeof(float2) * ng));
   T9_CUDA(cudaMalloc(&P.qfx, sizeof(long long) * ng));
   T9_CUDA(cudaMemset(P.qfx, 0, sizeof(long long) * ng));
   // the second grid: the induced-dipole half of the reciprocal forces runs
   // beside the permanent half
   T9_CUDA(cudaMalloc(&P.qgrid2, sizeof(float2) * ng));
   T9_CUDA(cudaMalloc(&P.qfx2, sizeof(long long) * ng));
   T9_CUDA(cudaMemset(P.qfx2, 0, sizeof(long long) * ng));
   // influence function in double precision, stored as float
   std::vector<double> m1, m2, m3;
   bspline_moduli(P.n1, c.bsorder, m1);
   bspline_moduli(P.n2, c.bsorder, m2);
   bspline_moduli(P.n3, c.bsorder, m3);
   const double pi = 3.14159265358979323846;
   const double pterm = (pi / c.aewald) * (pi / c.aewald);
   const double vol = c.box[0] * c.box[1] * c.box[2];
   std::vector<float> infl(ng);
   for (int k3 = 0; k3 < P.n3; ++k3)
      for (int k2 = 0; k2 < P.n2; ++k2)
         for (int k1 = 0; k1 < P.n1; ++k1) {
            size_t i = ((size_t)k3 * P.n2 + k2) * P.n1 + k1;
            int r1 = (k1 < (P.n1 + 1) / 2) ? k1 : k1 - P.n1;
            int r2 = (k2 < (P.n2 + 1) / 2) ? k2 : k2 - P.n2;
            int r3 = (k3 < (P.n3 + 1) / 2) ? k3 : k3 - P.n3;
            double h1 = r1 / c.box[0], h2 = r2 / c.box[1], h3 = r3 / c.box[2];
            double hsq = h1 * h1 + h2 * h2 + h3 * h3;
            double term = -pterm * hsq;
            double e = 0;
            if (i != 0 && term > -50)
               e = std::exp(term) / (hsq * pi * vol * m1[k1] * m2[k2] * m3[k3]);
            infl[i] = (float)e;
         }
   T9_CUDA(cudaMalloc(&P.org, sizeof(int4) * ctx->npad));
   T9_CUDA(cudaMalloc(&P.spl_lo, sizeof(float) * SPL_ROW * (size_t)ctx->npad));
   T9_CUDA(cudaMalloc(&P.spl_hi, sizeof(float) * SPL_ROW * (size_t)ctx->npad));
   float* d_infl = nullptr;
   T9_CUDA(cudaMalloc(&d_infl, sizeof(float) * ng));
   T9_CUDA(cudaMemcpy(d_infl, infl.data(), sizeof(float) * ng, cudaMemcpyHostToDevice));
   P.infl = d_infl;
   T9_CUDA(cudaMalloc(&P.fft_err, sizeof(int)));
   T9_CUDA(cudaMemset(P.fft_err, 0, sizeof(int)));
   if (cufftPlan3d(&P.plan, P.n3, P.n2, P.n1, CUFFT_C2C) != CUFFT_SUCCESS ||
      cufftPlan3d(&P.plan2, P.n3, P.n2, P.n1, CUFFT_C2C) != CUFFT_SUCCESS) {
      ctx->last_error = "cufftPlan3d failed";
      return T9GB_CUDA_ERR;
   }
   // the fused FFT: cubic grids of 32, 64 or 128 points per edge
   P.own_fft_ok = P.n1 == P.n2 && P.n2 == P.n3 && (P.n1 == 32 || P.n1 == 64 || P.n1 == 128);
   T9_CHECK(small_fft_setup(ctx));
   pme_choose(P, -1, 0);
   if (P.own_fft_ok) {
      if (P.n1 == 32)
         T9_CHECK(fft_setup_kernels<32>(ctx));
      else if (P.n1 == 64)
         T9_CHECK(fft_setup_kernels<64>(ctx));
      else
         T9_CHECK(fft_setup_kernels<128>(ctx));
      float2 tw[128];
      for (int k = 0; k < 128; ++k)
         tw[k] = make_float2((float)std::cos(2 * pi * k / 128.0), (float)-std::sin(2 * pi * k / 128.0));
      T9_CUDA(cudaMemcpyToSymbol(c_tw, tw, sizeof(tw)));
      T9_CUDA(cudaDeviceSynchronize());
   }
   return T9GB_OK;
}

// The fused transform is the default where it measured faster than cuFFT on
// GB300 (64^3: 0.627 vs 0.634 ms per induce step in the graph; at 128^3 cuFFT
// is faster); the one-cluster transform where it has a kernel and nothing else
// was asked for.  Every choice can be taken back.
bool pme_choose(PmeGrid& P, int choice, int fft_cl)
{
   const bool own = choice < 0 ? P.own_fft_ok && P.n1 <= 64 : choice != 0;
   const bool small = P.small_tw && choice < 0 && fft_cl == 0;
   const bool changed = own != P.own_fft || small != P.small_fft || fft_cl != P.fft_cl;
   P.choice = choice;
   P.fft_cl = fft_cl;
   P.own_fft = own;
   P.small_fft = small;
   return changed;
}

void pme_free(Context* ctx)
{
   PmeGrid& P = ctx->pme;
   if (P.plan)
      cufftDestroy(P.plan);
   if (P.plan2)
      cufftDestroy(P.plan2);
   cudaFree(P.qgrid2);
   cudaFree(P.qfx2);
   cudaFree(P.qgrid);
   cudaFree(P.qfx);
   cudaFree(P.infl);
   cudaFree(P.org);
   cudaFree(P.spl_lo);
   cudaFree(P.spl_hi);
   cudaFree(P.qstash);
   cudaFree(P.fft_err);
   cudaFree(P.small_tw);
   P = PmeGrid();
}

static Sites sites(const Context* ctx) { return Sites{ctx->pme.org, ctx->pme.spl_lo, ctx->pme.spl_hi}; }

static GridParams grid_params(const Context* ctx)
{
   const t9gb_config& c = ctx->cfg;
   GridParams G;
   G.n1 = c.nfft[0];
   G.n2 = c.nfft[1];
   G.n3 = c.nfft[2];
   G.r1 = (float)(1.0 / c.box[0]);
   G.r2 = (float)(1.0 / c.box[1]);
   G.r3 = (float)(1.0 / c.box[2]);
   G.a1 = (float)(c.nfft[0] / c.box[0]);
   G.a2 = (float)(c.nfft[1] / c.box[1]);
   G.a3 = (float)(c.nfft[2] / c.box[2]);
   G.selfterm = (float)(4.0 * c.aewald * c.aewald * c.aewald / (3.0 * 1.77245385090551602730));
   G.pk_s = (float)(1 << ctx->pme.pack_shift);
   G.pk_lim = (float)(1 << (31 - 5 - ctx->pme.pack_shift));
   G.range = ctx->status + (ctx->pme.probe ? ST_RANGE_L : ST_RANGE);
   return G;
}

static int conv_virial(Context* ctx, int vir, float wE, float wP, bool stash, double* out)
{
   PmeGrid& P = ctx->pme;
   const size_t ng = (size_t)P.n1 * P.n2 * P.n3;
   const t9gb_config& c = ctx->cfg;
   const float pterm = (float)((3.14159265358979323846 / c.aewald) * (3.14159265358979323846 / c.aewald));
   if ((stash || vir == 2) && !P.qstash)
      T9_CUDA(cudaMalloc(&P.qstash, sizeof(float2) * ng));
   const int vb = (int)std::min<size_t>((ng + 255) / 256, RED_MAX);
   if (vir == 1)
      k_conv_virial<1><<<vb, 256, 0, ctx->stream>>>(P.n1, P.n2, P.n3, (float)c.box[0], (float)c.box[1],
         (float)c.box[2], pterm, P.infl, P.qgrid, stash ? P.qstash : nullptr, wE, wP, ctx->red, out, ctx->status);
   else
      k_conv_virial<2><<<vb, 256, 0, ctx->stream>>>(P.n1, P.n2, P.n3, (float)c.box[0], (float)c.box[1],
         (float)c.box[2], pterm, P.infl, P.qgrid, P.qstash, wE, wP, ctx->red, out, ctx->status);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

// vir: 0 none, 1 permanent-grid k-space virial (wE, stash), 2 dipole-grid
// cross terms (wP); the sums go to out[0..6)
static int fft_conv(Context* ctx, int vir = 0, float wE = 0.f, float wP = 0.f, bool stash = false,
   double* out = nullptr)
{
   PmeGrid& P = ctx->pme;
   const size_t ng = (size_t)P.n1 * P.n2 * P.n3;
   const int cb = (int)std::min<size_t>((ng + 255) / 256, 152 * 16);
   prof_begin(ctx, P_FFT_CONV);
   int* range = ctx->status + (P.probe ? ST_RANGE_L : ST_RANGE);
   // while the learned guess trains, the transform that its weights were trained
   // with: AdamW's first steps divide by the size of a gradient, so a weight
   // of a small one follows the rounding of the dipoles (2.3e-5 of the weights
   // of 954 atoms between the two transforms, the dipoles 5e-7)
   if (P.small_fft && !vir && !(ctx->learn_mode & 1)) {
      T9_CHECK(launch_small_fft(ctx, range));
      prof_end(ctx);
      return T9GB_OK;
   }
   if (P.own_fft) {
      cudaStream_t st = ctx->stream;
      const bool split = vir != 0;
      const bool pdl = use_pdl(ctx);
      if (P.n1 == 32)
         fft_own_forward<32>(P, st, split, pdl, range);
      else if (P.n1 == 64)
         fft_own_forward<64>(P, st, split, pdl, range);
      else
         fft_own_forward<128>(P, st, split, pdl, range);
      if (split) {
         T9_CHECK(conv_virial(ctx, vir, wE, wP, stash, out));
         k_conv<<<cb, 256, 0, st>>>(ng, P.infl, P.qgrid);
      }
      if (P.n1 == 32)
         fft_own_inverse<32>(P, st, split, pdl && !split);
      else if (P.n1 == 64)
         fft_own_inverse<64>(P, st, split, pdl && !split);
      else
         fft_own_inverse<128>(P, st, split, pdl && !split);
      T9_CUDA(cudaGetLastError());
      prof_end(ctx);
      return T9GB_OK;
   }
   k_fx_to_grid<<<cb, 256, 0, ctx->stream>>>(ng, P.qfx, P.qgrid, P.packed ? 1 : 0,
      1.0f / (float)(1 << P.pack_shift), range);
   T9_CUDA(cudaGetLastError());
   cufftSetStream(P.plan, ctx->stream);
   if (cufftExecC2C(P.plan, (cufftComplex*)P.qgrid, (cufftComplex*)P.qgrid, CUFFT_FORWARD) != CUFFT_SUCCESS) {
      ctx->last_error = "cufftExecC2C forward failed";
      return T9GB_CUDA_ERR;
   }
   if (vir)
      T9_CHECK(conv_virial(ctx, vir, wE, wP, stash, out));
   k_conv<<<cb, 256, 0, ctx->stream>>>(ng, P.infl, P.qgrid);
   T9_CUDA(cudaGetLastError());
   if (cufftExecC2C(P.plan, (cufftComplex*)P.qgrid, (cufftComplex*)P.qgrid, CUFFT_INVERSE) != CUFFT_SUCCESS) {
      ctx->last_error = "cufftExecC2C inverse failed";
      return T9GB_CUDA_ERR;
   }
   prof_end(ctx);
   return T9GB_OK;
}

// Reciprocal permanent field in two halves: the grid (spread + transform,
// on ctx->stream) and the gather (recip + self into out6; acc: added to the
// real-space field stored there)
int launch_dfield_recip_grid(Context* ctx)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   prof_begin(ctx, P_SPREAD_MPOLE);
   ctx->pme.packed = false;
   k_spread<0><<<grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->srpole,
      nullptr, nullptr, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), nullptr);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return fft_conv(ctx);
}

int launch_dfield_recip_gather(Context* ctx, float* out6, bool acc)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   const int nb = grid_for((long long)ctx->n * 32, 256);
   prof_begin(ctx, P_GATHER_MPOLE);
   if (acc)
      k_gather_field<0, true><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->pme.qgrid, ctx->srpole, nullptr,
         out6, PcgAp{});
   else
      k_gather_field<0, false><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->pme.qgrid, ctx->srpole,
         nullptr, out6, PcgAp{});
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_dfield_recip(Context* ctx, float* out6)
{
   T9_CHECK(launch_dfield_recip_grid(ctx));
   return launch_dfield_recip_gather(ctx, out6, false);
}

int launch_ufield_recip_grid(Context* ctx, const float* u6)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   prof_begin(ctx, P_SPREAD_UIND);
   ctx->pme.packed = true;
   T9_CUDA(launch_k(use_pdl(ctx), k_spread<1, false>, grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream,
      ctx->n, G, sites(ctx), u6, nullptr, nullptr, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), nullptr));
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return fft_conv(ctx);
}

int launch_ufield_recip_gather(Context* ctx, const float* u6, float* out6, bool acc)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   const int nb = grid_for((long long)ctx->n * 32, 256);
   prof_begin(ctx, P_GATHER_UIND);
   T9_CUDA(launch_k(use_pdl(ctx), acc ? k_gather_field<1, true> : k_gather_field<1, false>, nb, 256, 0, ctx->stream,
      ctx->n, G, sites(ctx), ctx->pme.qgrid, nullptr, u6, out6, PcgAp{}));
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_ufield_recip(Context* ctx, const float* u6, float* out6)
{
   T9_CHECK(launch_ufield_recip_grid(ctx, u6));
   return launch_ufield_recip_gather(ctx, u6, out6, false);
}

static void swap_grids(PmeGrid& P)
{
   std::swap(P.qfx, P.qfx2);
   std::swap(P.qgrid, P.qgrid2);
   std::swap(P.plan, P.plan2);
}

int launch_ufield_recip_grid_alt(Context* ctx, const float* u6)
{
   swap_grids(ctx->pme);
   const int rc = launch_ufield_recip_grid(ctx, u6);
   swap_grids(ctx->pme);
   return rc;
}

int launch_ufield_recip_gather_alt(Context* ctx, const float* u6, float* out6)
{
   swap_grids(ctx->pme);
   const int rc = launch_ufield_recip_gather(ctx, u6, out6, true);
   swap_grids(ctx->pme);
   return rc;
}

// the CG search direction's grid: p = z + b p_old formed by the spread
int launch_ufield_recip_grid_dir(Context* ctx, const float* p6, const float* z6, const double* scal)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   prof_begin(ctx, P_SPREAD_UIND);
   ctx->pme.packed = true;
   T9_CUDA(launch_k(use_pdl(ctx), k_spread<1, true>, grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream,
      ctx->n, G, sites(ctx), p6, z6, scal, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), nullptr));
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return fft_conv(ctx);
}

// the CG search direction p = z + b p_old formed, stored in p6 and spread; its
// transform
int launch_ufield_spread_dir(Context* ctx, float* p6, const float* z6, const double* scal)
{
   GridParams G = grid_params(ctx);
   ctx->pme.packed = true;
   T9_CUDA(launch_k(use_pdl(ctx), k_spread<1, true>, grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream,
      ctx->n, G, sites(ctx), p6, z6, scal, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), p6));
   return T9GB_OK;
}

int launch_ufield_transform(Context* ctx) { return fft_conv(ctx); }

// recip + self field of the search direction p = z + b p_old (P.conj =
// p_old, P.zrsd = z, P.scal = b) added to the real-space field in out6
int launch_ufield_recip_gather_dir(Context* ctx, float* out6, const PcgAp& P)
{
   GridParams G = grid_params(ctx);
   const int nb = grid_for((long long)ctx->n * 32, 256);
   prof_begin(ctx, P_GATHER_UIND);
   k_gather_field<1, true, false, true><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->pme.qgrid, nullptr,
      nullptr, out6, P);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

// recip + self field of the search direction added to the real-space field
// in out6, then p, Ap and the step length (PcgAp)
int launch_ufield_recip_gather_ap(Context* ctx, float* out6, const PcgAp& P)
{
   GridParams G = grid_params(ctx);
   const int nb = std::min(RED_MAX, grid_for((long long)ctx->n * 32, 256));
   prof_begin(ctx, P_GATHER_UIND);
   k_gather_field<1, true, true><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->pme.qgrid, nullptr, nullptr,
      out6, P);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

}  // namespace t9gb

namespace t9gb {
int launch_empole_recip(Context* ctx, double* e_atom)
{
   if (!ctx->cfg.use_ewald)
      return T9GB_OK;
   GridParams G = grid_params(ctx);
   ctx->pme.packed = false;
   k_spread<0><<<grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->srpole,
      nullptr, nullptr, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), nullptr);
   T9_CUDA(cudaGetLastError());
   T9_CHECK(fft_conv(ctx));
   k_empole_recip_self<<<grid_for((long long)ctx->n * 32, 256), 256, 0, ctx->stream>>>(ctx->n, G,
      (float)ctx->cfg.electric, (float)ctx->cfg.aewald, ctx->spos, ctx->pme.qgrid, ctx->srpole, e_atom,
      e_atom + ctx->npad);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}
}  // namespace t9gb

namespace t9gb {
// Atoms per warp of the force gathers: eight where that still gives an SM 20
// warps, four below, one where four leave most of the chip idle (both
// kernels, us at one / four atoms: 648 atoms 15 / 23, 3,000 17 / 24, 5,184
// 24 / 25, 8,232 29 / 26)
static int force_atoms(int n) { return n > 24576 ? 8 : (n > 6144 ? 4 : 1); }

// a kernel by that number
#define T9_FORCE_ATOMS(FA, KERNEL, ...)                                                                                \
   ((FA) == 8 ? KERNEL<__VA_ARGS__ 8> : (FA) == 4 ? KERNEL<__VA_ARGS__ 4> : KERNEL<__VA_ARGS__ 1>)

// reciprocal forces for elec_forces (force.cu), in two halves: the
// permanent-multipole grid (forces and torque fields of the multipoles, the
// induced dipoles' force in the permanent field) and the induced-dipole
// grid.  wrec (may be null): the per-slot fractional-transform virial rows,
// k-space sums in scal[40..52); with the virial the dipole half reads the
// permanent half's transformed grid, so the two run in order.
int launch_force_recip_perm(Context* ctx, bool mpole, bool polar, float* wrec)
{
   GridParams G = grid_params(ctx);
   const int nb = grid_for((long long)ctx->n * 32, 256);
   const int np = ctx->npad;
   const float f = (float)ctx->cfg.electric, a = (float)ctx->cfg.aewald;
   const bool vir = wrec != nullptr;
   if (vir) {
      T9_CUDA(cudaMemsetAsync(wrec, 0, sizeof(float) * 9 * np, ctx->stream));
      T9_CUDA(cudaMemsetAsync(ctx->scal + 40, 0, sizeof(double) * 12, ctx->stream));
   }
   ctx->pme.packed = false;
   k_spread<0><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->srpole,
      nullptr, nullptr, reinterpret_cast<unsigned long long*>(ctx->pme.qfx), nullptr);
   T9_CUDA(cudaGetLastError());
   T9_CHECK(fft_conv(ctx, vir ? 1 : 0, mpole ? 0.5f * f : 0.f, 0.f, vir && polar, ctx->scal + 40));
   double* er = ctx->e_atom + np;
   double* es = ctx->e_atom + 2 * np;
   const int fa = force_atoms(ctx->n), fb = grid_for(ctx->n, FORCE_WARPS * fa);
   auto k = mpole && polar ? T9_FORCE_ATOMS(fa, k_gather_force_perm, true, true, )
      : mpole              ? T9_FORCE_ATOMS(fa, k_gather_force_perm, true, false, )
                           : T9_FORCE_ATOMS(fa, k_gather_force_perm, false, true, );
   k<<<fb, 32 * FORCE_WARPS, 0, ctx->stream>>>(ctx->n, np, G, f, a, sites(ctx), ctx->pme.qgrid, ctx->srpole, ctx->uind,
      ctx->frecp, ctx->trecp, mpole ? er : nullptr, mpole ? es : nullptr, wrec);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

// alt: on the second grid (and FFT plan), so that it can run beside the
// permanent half on another stream (no virial)
int launch_force_recip_uind(Context* ctx, float* wrec, bool alt)
{
   PmeGrid& P = ctx->pme;
   if (alt) {
      std::swap(P.qfx, P.qfx2);
      std::swap(P.qgrid, P.qgrid2);
      std::swap(P.plan, P.plan2);
   }
   GridParams G = grid_params(ctx);
   const int nb = grid_for((long long)ctx->n * 32, 256);
   const float f = (float)ctx->cfg.electric;
   const bool vir = wrec != nullptr;
   P.packed = true;
   k_spread<1><<<nb, 256, 0, ctx->stream>>>(ctx->n, G, sites(ctx), ctx->uind,
      nullptr, nullptr, reinterpret_cast<unsigned long long*>(P.qfx), nullptr);
   int rc = cudaGetLastError() == cudaSuccess ? T9GB_OK : T9GB_CUDA_ERR;
   if (rc == T9GB_OK)
      rc = fft_conv(ctx, vir ? 2 : 0, 0.f, 0.5f * f, false, ctx->scal + 46);
   if (rc == T9GB_OK) {
      const int fa = force_atoms(ctx->n);
      auto k = T9_FORCE_ATOMS(fa, k_gather_force_uind);
      k<<<grid_for(ctx->n, FORCE_WARPS * fa), 32 * FORCE_WARPS, 0, ctx->stream>>>(ctx->n, ctx->npad, G, f, sites(ctx),
         P.qgrid, ctx->srpole, ctx->uind, ctx->frecu, ctx->trecu, wrec);
      if (cudaGetLastError() != cudaSuccess)
         rc = T9GB_CUDA_ERR;
   }
   if (alt) {
      std::swap(P.qfx, P.qfx2);
      std::swap(P.qgrid, P.qgrid2);
      std::swap(P.plan, P.plan2);
   }
   return rc;
}

int launch_force_recip(Context* ctx, bool mpole, bool polar, float* wrec)
{
   T9_CHECK(launch_force_recip_perm(ctx, mpole, polar, wrec));
   if (polar)
      T9_CHECK(launch_force_recip_uind(ctx, wrec, false));
   return T9GB_OK;
}
}  // namespace t9gb
