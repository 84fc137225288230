// Real-space pair kernels over the per-step neighbour list.
//
// G consecutive lanes own one atom i (t9gb_pair_lanes: 16 up to 768 atoms, 8 up to 32,768,
// 4 above): lane g walks the list entries g, g+G, g+2G, ... of atom i
// (consecutive addresses per step, two entries in flight per trip), then the
// scaled partners of i the same way; the partial fields are combined with a
// fixed xor-shuffle tree and written with plain stores.  Every pair is
// evaluated from both sides (full list), so no atomics are needed and each
// field component is a sum in a fixed order: results are bit-reproducible.
// 12,288 atoms at 8 lanes give 98,304 threads, ~20 warps on each of the 152
// SMs.
//
// Pair arithmetic restates the reference's pair_dfield_v2 / pair_ufield_v2
// (include/seq/pair_field.h:127-256, :333-420) for the atom-i side, Thole
// damping damp_thole2/3 (include/seq/damp.h:8-44), the Ewald b_n recursion
// damp_ewald (include/seq/damp.h:136-151), and the preconditioner pair of
// sparsePrecond_cu1 (src/cu/amoeba/sparsePrecond_cu1.cc:60-120).  The k side
// of the reference's pair functions equals the i-side formula evaluated from
// atom k with the separation reversed, which is what the full list does.
#include "pair.cuh"
#include "reduce.cuh"

namespace t9gb {


__device__ __forceinline__ void thole_damp(float r, float pdi, float pgamma, float pdk, float& s3, float& s5,
   float& s7)
{
   float damp = pdi * pdk;
   float ratio = r * __frcp_rn(damp);
   damp = (damp == 0.f) ? -1.0e16f : -pgamma * ratio * ratio * ratio;
   float ex = __expf(damp);
   s3 = 1.f - ex;
   s5 = 1.f - ex * (1.f - damp);
   s7 = 1.f - ex * (1.f - damp + 0.6f * damp * damp);
}

__device__ __forceinline__ void ewald_bn(const PairParams& P, float r, float invr, float rr2, float& b1, float& b2,
   float& b3)
{
   float ralpha = P.aewald * r;
   float exp2a = __expf(-ralpha * ralpha);
   float b0 = erfc_hastings(ralpha, exp2a) * invr;
   b1 = (b0 + P.ec1 * exp2a) * rr2;
   b2 = (3.f * b1 + P.ec2 * exp2a) * rr2;
   b3 = (5.f * b2 + P.ec3 * exp2a) * rr2;
}




__device__ __forceinline__ float pick6(const float* f, int g)
{
   float v = f[0];
#pragma unroll
   for (int c = 1; c < 6; ++c)
      if (g == c)
         v = f[c];
   return v;
}

// The six sums of a group of G lanes: fn(c, sum) for the components c = g,
// g + G, ... < 6 that lane g of the group finishes.  Sums in the order of an
// xor tree, farthest lanes first; for G = 8 by the halving tree (the same
// additions in 7 shuffles where six trees take 18).
template <int G, class F>
__device__ __forceinline__ void for_own6(float* f, F&& fn)
{
   const int lane = threadIdx.x & 31, g = lane & (G - 1);
   if constexpr (G == 8) {
      const float v = warp_sums<6, 4>(f, lane);
      // components 0-2 sit in lanes 0-2 of the group, 3-5 in lanes 4-6
      const float w = __shfl_sync(0xffffffffu, v, (lane & 24) | (g < 3 ? g : (g + 1) & 7));
      if (g < 6)
         fn(g, w);
   } else {
      group_reduce<G, 6>(f);
#pragma unroll
      for (int c0 = 0; c0 < 6; c0 += G) {
         const int c = c0 + g;
         if (c < 6)
            fn(c, pick6(f, c));
      }
   }
}

// ---------------------------------------------------------------------------
// Dipole tensor rows.  The mutual field -T u (pair_ufield_v2) and the sparse
// preconditioner's off-diagonal part have one form,
//   f_i = sum_k [ c2 (d . v_k) d - c1 v_k ],  d = r_k - r_i,
// and their radial factors (c1, c2) depend on the positions only: the filter
// forms them once per position update for every listed pair, and a solve of
// m iterations reads them 2 m + 2 times.  A pair then costs an index, 8 bytes
// of factors, one position and one row, and about 40 instructions (the
// kernels that formed the factors in place spent 168 per pair and waited on
// the transcendental chain).  The sub-lists and factors are stored by tiles of
// 32 / G atoms (ListView), so that a warp's index load is one 128-byte line
// and its factor load two; the neighbour's row is one 32-byte load.  What
// bounds the rows is the L1's rate of one line per cycle (1 + 2 + 11 + 14 lines
// for 32 pairs, 47 before; from cold caches ncu has the L1 at 68 and 75 % for
// the mutual field and the preconditioner of 98,304 atoms, 4 lanes).  GB300,
// ncu, 12,288 / 98,304 atoms: mutual field 20.6 -> 16.2 / 97 -> 77 us,
// preconditioner 20.5 -> 16.0 / 82 -> 63, permanent field 26.3 -> 19.1 /
// 120 -> 96, filter 23 -> 31 / 118 -> 205 (once per position update).

// a sub-list with its factors, tiled (ListView) for the kernels' lane count:
// counts per slot, indices, factors, and the factors of the scaled partners
struct TensorList {
   const int *nbr, *cnt;
   const float2 *coef, *spc;
};

// scaled partners of every slot (CSR)
struct Partners {
   const int *start, *j;
};

// slot i's first entry in a tiled list of G lanes per atom
template <int G>
__device__ __forceinline__ size_t tile_at(int cap, int i)
{
   constexpr int W = 32 / G;
   return (size_t)(i / W) * W * cap + (i % W) * G;
}

__device__ __forceinline__ void tensor_add(float3 d, float2 c, const float* v, float* f)
{
   float q = c.y * (d.x * v[0] + d.y * v[1] + d.z * v[2]);
   f[0] += q * d.x - c.x * v[0];
   f[1] += q * d.y - c.x * v[1];
   f[2] += q * d.z - c.x * v[2];
   q = c.y * (d.x * v[3] + d.y * v[4] + d.z * v[5]);
   f[3] += q * d.x - c.x * v[3];
   f[4] += q * d.y - c.x * v[4];
   f[5] += q * d.z - c.x * v[5];
}

// list entries and factors: read once per application, kept out of L1 so
// that the neighbours' positions and rows stay there
__device__ __forceinline__ int stream_index(const int* p)
{
   int v;
   asm volatile("ld.global.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
   return v;
}

__device__ __forceinline__ int stream_index(const unsigned short* p) { return *p; }

__device__ __forceinline__ float2 stream_coef(const float2* p)
{
   float2 v;
   asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
   return v;
}

// neighbour j's position and row from global memory; DIR: the row is the CG
// search direction p = z + b p_old, formed as it is read
template <bool DIR>
struct GlobalRows {
   const float4* spos;
   const float *u8, *z8;
   float bd, bp;
   __device__ __forceinline__ void get(int j, float4& p, float* v) const
   {
      p = spos[j];
      if (DIR)
         dir_row(u8, z8, j, bd, bp, v);
      else
         load8_wide(u8, j, v);
   }
};

// the row sum of one atom's lane g of G: U entries per trip, their loads in
// flight together and added in order, the next trip's indices loaded ahead.
// ip, cp: the lane's first index and factors; is: index stride from one entry
// of the lane to the next (factors: 32).
template <int G, int U, class IDX, class R>
__device__ __forceinline__ void tensor_row(const PairParams& P, const IDX* __restrict__ ip, int is,
   const float2* __restrict__ cp, int cnt, int g, float4 pi, const R& rows, float* f)
{
   int j[U];
#pragma unroll
   for (int q = 0; q < U; ++q)
      j[q] = g + q * G < cnt ? stream_index(ip + q * is) : -1;
   for (int k = g; k < cnt; k += U * G) {
      float2 c[U];
      float4 p[U];
      float u[U][8];
#pragma unroll
      for (int q = 0; q < U; ++q)
         if (q == 0 || j[q] >= 0) {
            c[q] = stream_coef(cp + 32 * q);
            rows.get(j[q], p[q], u[q]);
         }
      ip += U * is;
      cp += 32 * U;
      int n[U];
#pragma unroll
      for (int q = 0; q < U; ++q)
         n[q] = k + (U + q) * G < cnt ? stream_index(ip + q * is) : -1;
#pragma unroll
      for (int q = 0; q < U; ++q) {
         if (q == 0 || j[q] >= 0)
            tensor_add(sep(P, pi, p[q]), c[q], u[q], f);
         j[q] = n[q];
      }
   }
}

// the scaled partners of slot i (their factors are zero beyond the cutoff)
template <int G, class R>
__device__ __forceinline__ void tensor_partners(const PairParams& P, const Partners& S, const float2* __restrict__ spc,
   int i, int g, float4 pi, const R& rows, float* f)
{
   const int pa = S.start[i], pb = S.start[i + 1];
   for (int q = pa + g; q < pb; q += G) {
      const float2 c = spc[q];
      float4 p;
      float u[8];
      rows.get(S.j[q], p, u);
      tensor_add(sep(P, pi, p), c, u, f);
   }
}

// both, from global memory
template <int G, int U, class R>
__device__ __forceinline__ void tensor_sum(const PairParams& P, const TensorList& T, const Partners& S, int i, int g,
   const float4* __restrict__ spos, const R& rows, float* f)
{
   const float4 pi = spos[i];
   const size_t at = tile_at<G>(P.cap, i) + g;
   tensor_row<G, U>(P, T.nbr + at, 32, T.coef + at, T.cnt[i], g, pi, rows, f);
   tensor_partners<G>(P, S, T.spc, i, g, pi, rows, f);
}

template <int G, bool DIR, int U = 2>
__global__ void __launch_bounds__(256) k_ufield_real(PairParams P, int npad, TensorList T, Partners S,
   const float4* __restrict__ spos, const float* __restrict__ u8, const float* __restrict__ z8,
   const double* __restrict__ scal, const float* __restrict__ base8, float* __restrict__ out8)
{
   const int tid = blockIdx.x * blockDim.x + threadIdx.x;
   const int i = tid / G, g = tid % G;
   if (i >= npad)
      return;
   pdl_wait();
   float f[6] = {0, 0, 0, 0, 0, 0};
   if (i < P.n) {
      GlobalRows<DIR> rows{spos, u8, z8, 0.f, 0.f};
      if (DIR) {
         rows.bd = (float)scal[S_B_D];
         rows.bp = (float)scal[S_B_P];
      }
      tensor_sum<G, U>(P, T, S, i, g, spos, rows, f);
   }
   pdl_trigger();
   for_own6<G>(f, [&](int c, float v) { out8[8 * i + c] = base8 && i < P.n ? v + base8[8 * i + c] : v; });
}

// ---------------------------------------------------------------------------
// permanent field, i side (pair_dfield_v2)

__device__ __forceinline__ void dfield_i(const PairParams& P, float r2, float3 d, float dscale, float pscale,
   float pdi, float pti, float pdk, float ptk, const float* mk, float* f)
{
   float invr = rsqrtf(r2);
   float r = r2 * invr;
   float rr2 = invr * invr;
   float rr3 = invr * rr2;
   float rr5 = 3.f * rr3 * rr2;
   float rr7 = 5.f * rr5 * rr2;
   float s3, s5, s7;
   thole_damp(r, pdi, pair_gamma(P, pti, ptk), pdk, s3, s5, s7);
   float e1 = 0.f, e2 = 0.f, e3 = 0.f;
   if (P.ewald)
      ewald_bn(P, r, invr, rr2, e1, e2, e3);
   // mk: c, dx, dy, dz, qxx, qyy, qzz, qxy, qxz, qyz
   const float dkr = mk[1] * d.x + mk[2] * d.y + mk[3] * d.z;
   const float qkx = mk[4] * d.x + mk[7] * d.y + mk[8] * d.z;
   const float qky = mk[7] * d.x + mk[5] * d.y + mk[9] * d.z;
   const float qkz = mk[8] * d.x + mk[9] * d.y + mk[6] * d.z;
   const float qkr = qkx * d.x + qky * d.y + qkz * d.z;
   float b1, b2, b3;
   if (P.ewald) {
      b1 = e1 - (1.f - dscale * s3) * rr3;
      b2 = e2 - (1.f - dscale * s5) * rr5;
      b3 = e3 - (1.f - dscale * s7) * rr7;
   } else {
      b1 = dscale * s3 * rr3;
      b2 = dscale * s5 * rr5;
      b3 = dscale * s7 * rr7;
   }
   float c1 = -(b1 * mk[0] - b2 * dkr + b3 * qkr);
   float fx = c1 * d.x - b1 * mk[1] + 2.f * b2 * qkx;
   float fy = c1 * d.y - b1 * mk[2] + 2.f * b2 * qky;
   float fz = c1 * d.z - b1 * mk[3] + 2.f * b2 * qkz;
   f[0] += fx;
   f[1] += fy;
   f[2] += fz;
   if (pscale != dscale) {
      if (P.ewald) {
         b1 = e1 - (1.f - pscale * s3) * rr3;
         b2 = e2 - (1.f - pscale * s5) * rr5;
         b3 = e3 - (1.f - pscale * s7) * rr7;
      } else {
         b1 = pscale * s3 * rr3;
         b2 = pscale * s5 * rr5;
         b3 = pscale * s7 * rr7;
      }
      c1 = -(b1 * mk[0] - b2 * dkr + b3 * qkr);
      fx = c1 * d.x - b1 * mk[1] + 2.f * b2 * qkx;
      fy = c1 * d.y - b1 * mk[2] + 2.f * b2 * qky;
      fz = c1 * d.z - b1 * mk[3] + 2.f * b2 * qkz;
   }
   f[3] += fx;
   f[4] += fy;
   f[5] += fz;
}

// one 48-byte multipole row: q, d xyz, qxx, qyy, qzz, qxy, qxz, qyz, thole, polarizability
__device__ __forceinline__ void load12(const float* __restrict__ rp, int s, float* m)
{
   const float4* p = reinterpret_cast<const float4*>(rp + 12 * s);
#pragma unroll
   for (int c = 0; c < 3; ++c) {
      const float4 v = p[c];
      m[4 * c] = v.x;
      m[4 * c + 1] = v.y;
      m[4 * c + 2] = v.z;
      m[4 * c + 3] = v.w;
   }
}

// the field of multipole row mk at separation d with radial factors b1-b3
__device__ __forceinline__ void mpole_field(float3 d, float b1, float b2, float b3, const float* mk, float* f)
{
   const float dkr = mk[1] * d.x + mk[2] * d.y + mk[3] * d.z;
   const float qkx = mk[4] * d.x + mk[7] * d.y + mk[8] * d.z;
   const float qky = mk[7] * d.x + mk[5] * d.y + mk[9] * d.z;
   const float qkz = mk[8] * d.x + mk[9] * d.y + mk[6] * d.z;
   const float qkr = qkx * d.x + qky * d.y + qkz * d.z;
   const float c1 = -(b1 * mk[0] - b2 * dkr + b3 * qkr);
   f[0] += c1 * d.x - b1 * mk[1] + 2.f * b2 * qkx;
   f[1] += c1 * d.y - b1 * mk[2] + 2.f * b2 * qky;
   f[2] += c1 * d.z - b1 * mk[3] + 2.f * b2 * qkz;
}

// the unscaled pairs, whose field is the same for both sets, with the
// filter's radial factors (T.coef: b1; coefd: b2, b3), then the scaled
// partners
template <int G>
__global__ void __launch_bounds__(256) k_dfield_real(PairParams P, int npad, TensorList T,
   const float2* __restrict__ coefd, const int* __restrict__ sp_start, const int* __restrict__ sp_j,
   const float4* __restrict__ sp_sc, const float4* __restrict__ spos, const float* __restrict__ rp,
   const float* __restrict__ base8, const float* __restrict__ exfld, float* __restrict__ out8)
{
   const int tid = blockIdx.x * blockDim.x + threadIdx.x;
   const int i = tid / G, g = tid % G;
   if (i >= npad)
      return;
   float f[6] = {0, 0, 0, 0, 0, 0};
   if (i < P.n) {
      const float4 pi = spos[i];
      const float pti = rp[12 * i + 10];
      size_t at = tile_at<G>(P.cap, i) + g;
      const int cnt = T.cnt[i];
      int j = g < cnt ? stream_index(T.nbr + at) : 0;
      for (int k = g; k < cnt; k += G) {
         const float b1 = stream_coef(T.coef + at).x;
         const float2 c = stream_coef(coefd + at);
         const float4 pk = spos[j];
         float mk[12];
         load12(rp, j, mk);
         at += 32;
         j = k + G < cnt ? stream_index(T.nbr + at) : 0;
         mpole_field(sep(P, pi, pk), b1, c.x, c.y, mk, f);
      }
      f[3] = f[0];
      f[4] = f[1];
      f[5] = f[2];
      const int pa = sp_start[i], pb = sp_start[i + 1];
      for (int q = pa + g; q < pb; q += G) {
         const int jq = sp_j[q];
         const float4 pk = spos[jq];
         const float3 d = sep(P, pi, pk);
         const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
         if (r2 <= P.cut2) {
            float mk[12];
            load12(rp, jq, mk);
            const float4 sc = sp_sc[q];
            dfield_i(P, r2, d, sc.y, sc.z, pi.w, pti, pk.w, mk[10], mk, f);
         }
      }
   }
   for_own6<G>(f, [&](int c, float v) {
      if (i < P.n) {
         // uniform external field on both sets (extfieldModifyDField_cu1,
         // src/cu/amoeba/empole.cu:139-159); zero when none is set
         v += exfld[c < 3 ? c : c - 3];
         if (base8)
            v += base8[8 * i + c];
      }
      out8[8 * i + c] = v;
   });
}

// ---------------------------------------------------------------------------
// sparse preconditioner: z_i = udiag alpha_i r_i + sum_k alpha_i alpha_k T_ik r_k,
// the filter's factors holding alpha_i alpha_k and the Thole damping

template <int G>
__global__ void __launch_bounds__(256) k_precond_sparse(PairParams P, int npad, float udiag,
   TensorList T, Partners S, const float4* __restrict__ spos, const float* __restrict__ r8, float* __restrict__ z8)
{
   const int tid = blockIdx.x * blockDim.x + threadIdx.x;
   const int i = tid / G, g = tid % G;
   if (i >= npad)
      return;
   float f[6] = {0, 0, 0, 0, 0, 0};
   if (i < P.n)
      tensor_sum<G, 2>(P, T, S, i, g, spos, GlobalRows<false>{spos, r8, nullptr, 0.f, 0.f}, f);
   const float poli = r8[8 * i + 7];
   for_own6<G>(f, [&](int c, float v) { z8[8 * i + c] = udiag * poli * r8[8 * i + c] + v; });
}

// z = M r of slot i from its row sums: stored, with the r.z and r.r sums
template <int G>
__device__ __forceinline__ void precond_store(int i, float udiag, float* f, const float* __restrict__ r8,
   float* __restrict__ z8, const PcgDots& D, float* dots)
{
   const float poli = r8[8 * i + 7];
   for_own6<G>(f, [&](int c, float v) {
      const float r = r8[8 * i + c];
      const float z = udiag * poli * r + v;
      z8[8 * i + c] = z;
      if (D.init)
         D.conj[8 * i + c] = z;
      if (c < 3) {
         dots[0] += r * z;
         dots[2] += r * r;
      } else {
         dots[1] += r * z;
         dots[3] += r * r;
      }
   });
}

// z = M r fused with the partial sums r.z, r.r (d and p) and, in the last
// block, the CG scalars.  Slots are visited block-strided, 256 / G per
// block per trip (npad is a multiple of 32, so every lane of a block makes
// the same trips); at most RED_MAX blocks.
template <int G, int U = 2>
__global__ void __launch_bounds__(256, U > 2 ? 2 : 4) k_precond_sparse_dots(PairParams P, int npad, float udiag,
   TensorList T, Partners S, const float4* __restrict__ spos, const float* __restrict__ r8, float* __restrict__ z8,
   PcgDots D)
{
   pdl_wait();
   __shared__ double sh[64];
   constexpr int PER = 256 / G;
   const int g = threadIdx.x % G;
   float dots[4] = {0.f, 0.f, 0.f, 0.f};
   const GlobalRows<false> rows{spos, r8, nullptr, 0.f, 0.f};
   for (int i = blockIdx.x * PER + threadIdx.x / G; i < npad; i += gridDim.x * PER) {
      float f[6] = {0, 0, 0, 0, 0, 0};
      if (i < P.n)
         tensor_sum<G, U>(P, T, S, i, g, spos, rows, f);
      precond_store<G>(i, udiag, f, r8, z8, D, dots);
   }
   pdl_trigger();
   store_partials_f<4>(D.red, R_RZ_D, dots, sh);
   if (!last_block(D.state + ST_TICKET0))
      return;
   double tot[4];
   sum_slots(D.red, R_RZ_D, 4, gridDim.x, sh, tot);
   if (threadIdx.x == 0)
      pcg_scalars(tot, D.scal, D.state, D.init, D.n, D.debye, D.poleps, D.politer, D.miniter, D.handle,
         D.use_handle);
}

// ---------------------------------------------------------------------------
// Staged field and preconditioner kernels (t9gb_pair_staging): one CTA per
// 32-slot block (32 atoms x G lanes).  The block's j-blocks (the 32-slot
// blocks its sub-list entries fall in, listed by the filter) are copied into
// shared memory by the bulk-copy engine (cp.async.bulk: one 512-byte
// position copy and one 1-KB row copy per j-block, completing on an
// mbarrier), and every neighbour row is then read from shared memory through
// the entry's local index: one coalesced 2-byte index load per neighbour
// instead of a dependent scattered 48-byte global gather.  The neighbour
// order and the arithmetic are those of the global-memory kernels, so the
// fields are bit-identical to theirs; a block with more j-blocks than
// STAGE_JB_CAP reads its rows from global memory the same way.

constexpr unsigned STAGE_POS_BYTES = 32 * 16;   // one j-block of positions
constexpr unsigned STAGE_ROW_BYTES = 32 * 32;   // one j-block of 8-float rows
constexpr size_t STAGE_SMEM = (size_t)STAGE_JB_CAP * (STAGE_POS_BYTES + STAGE_ROW_BYTES);

// Stages the j-blocks jl[0..cnt) of positions and rows and waits for them
// (phase `phase` of the CTA's mbarrier); a wait that runs out is recorded in
// *err.  The caller has synchronised the CTA since its last read of the
// staging buffers.
__device__ __forceinline__ void stage_rows(unsigned char* stg, unsigned bar, unsigned phase, const int* __restrict__ jl,
   int cnt, const float4* __restrict__ spos, const float* __restrict__ r8, int* __restrict__ err)
{
   const unsigned pos_s = (unsigned)__cvta_generic_to_shared(stg);
   const unsigned row_s = pos_s + STAGE_JB_CAP * STAGE_POS_BYTES;
   if (threadIdx.x == 0)
      mbar_expect_tx(bar, (unsigned)cnt * (STAGE_POS_BYTES + STAGE_ROW_BYTES));
   // the previous pass's reads of the buffers (generic proxy) before the
   // copies' writes (async proxy)
   asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
   for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
      const int jb = jl[q];
      bulk_g2s(pos_s + q * STAGE_POS_BYTES, spos + (size_t)jb * 32, STAGE_POS_BYTES, bar);
      bulk_g2s(row_s + q * STAGE_ROW_BYTES, r8 + (size_t)jb * 32 * 8, STAGE_ROW_BYTES, bar);
   }
   if (mbar_wait_bounded(bar, phase))
      return;
   if (threadIdx.x == 0)
      atomicExch(err, 1);
   mbar_wait_bounded(bar, phase);  // the copies in flight, before the buffers are reused
}

// neighbour rows from the staged buffers, by local index
struct StagedRows {
   const unsigned char* stg;
   __device__ __forceinline__ void get(int L, float4& p, float* v) const
   {
      p = reinterpret_cast<const float4*>(stg)[L];
      const float4* r = reinterpret_cast<const float4*>(stg + STAGE_JB_CAP * STAGE_POS_BYTES) + 2 * L;
      const float4 x = r[0], y = r[1];
      v[0] = x.x;
      v[1] = x.y;
      v[2] = x.z;
      v[3] = x.w;
      v[4] = y.x;
      v[5] = y.y;
      v[6] = y.z;
      v[7] = y.w;
   }
};

// the list from the staged rows (nbr_l: the row's local indices), the scaled
// partners from global memory
template <int G>
__device__ __forceinline__ void staged_sum(const PairParams& P, const TensorList& T, const Partners& S,
   const unsigned short* __restrict__ nbr_l, int i, int g, const float4* __restrict__ spos, const StagedRows& stg,
   const GlobalRows<false>& rows, float* f)
{
   const float4 pi = spos[i];
   tensor_row<G, 2>(P, nbr_l + (size_t)i * P.cap + g, G, T.coef + tile_at<G>(P.cap, i) + g, T.cnt[i], g, pi, stg, f);
   tensor_partners<G>(P, S, T.spc, i, g, pi, rows, f);
}

template <int G>
__global__ void __launch_bounds__(32 * G) k_ufield_stg(PairParams P, TensorList T, Partners S,
   const unsigned short* __restrict__ nbr_l, const int* __restrict__ jbl, const int* __restrict__ jbn,
   const float4* __restrict__ spos, const float* __restrict__ u8, const float* __restrict__ base8, float* __restrict__ out8, int* __restrict__ err)
{
   pdl_wait();
   extern __shared__ __align__(128) unsigned char stg[];
   __shared__ __align__(8) unsigned long long bar;
   const int blk = blockIdx.x;
   const int i = blk * 32 + threadIdx.x / G, g = threadIdx.x % G;
   const int nj = jbn[blk];
   const bool staged = nj <= STAGE_JB_CAP;
   if (staged) {
      const unsigned bar_s = (unsigned)__cvta_generic_to_shared(&bar);
      if (threadIdx.x == 0)
         mbar_init(bar_s, 1);
      __syncthreads();
      stage_rows(stg, bar_s, 0, jbl + (size_t)blk * STAGE_JB_CAP, nj, spos, u8, err);
   }
   float f[6] = {0, 0, 0, 0, 0, 0};
   const GlobalRows<false> rows{spos, u8, nullptr, 0.f, 0.f};
   if (i < P.n && staged)
      staged_sum<G>(P, T, S, nbr_l, i, g, spos, StagedRows{stg}, rows, f);
   else if (i < P.n)
      tensor_sum<G, 2>(P, T, S, i, g, spos, rows, f);
   pdl_trigger();
   for_own6<G>(f, [&](int c, float v) { out8[8 * i + c] = base8 && i < P.n ? base8[8 * i + c] + v : v; });
}

// z = M r with the r.z / r.r partial sums and, in the last block, the CG
// scalars (k_precond_sparse_dots), one 32-slot block per CTA pass; a CTA
// takes blocks blockIdx.x, + gridDim.x, ... (at most RED_MAX CTAs), the
// staging mbarrier's phase flipping with each staged pass.
template <int G>
__global__ void __launch_bounds__(32 * G) k_precond_dots_stg(PairParams P, int nblk, float udiag,
   TensorList T, Partners S, const unsigned short* __restrict__ nbr_l, const int* __restrict__ jbl,
   const int* __restrict__ jbn, const float4* __restrict__ spos, const float* __restrict__ r8, float* __restrict__ z8, PcgDots D,
   int* __restrict__ err)
{
   pdl_wait();
   extern __shared__ __align__(128) unsigned char stg[];
   __shared__ __align__(8) unsigned long long bar;
   __shared__ double sh[64];
   const unsigned bar_s = (unsigned)__cvta_generic_to_shared(&bar);
   if (threadIdx.x == 0)
      mbar_init(bar_s, 1);
   __syncthreads();
   const int g = threadIdx.x % G;
   float dots[4] = {0.f, 0.f, 0.f, 0.f};
   unsigned phase = 0;
   for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
      const int i = blk * 32 + threadIdx.x / G;
      const int nj = jbn[blk];
      const bool staged = nj <= STAGE_JB_CAP;
      if (staged) {
         __syncthreads();  // the previous pass has read the buffers
         stage_rows(stg, bar_s, phase, jbl + (size_t)blk * STAGE_JB_CAP, nj, spos, r8, err);
         phase ^= 1u;
      }
      float f[6] = {0, 0, 0, 0, 0, 0};
      const GlobalRows<false> rows{spos, r8, nullptr, 0.f, 0.f};
      if (i < P.n && staged)
         staged_sum<G>(P, T, S, nbr_l, i, g, spos, StagedRows{stg}, rows, f);
      else if (i < P.n)
         tensor_sum<G, 2>(P, T, S, i, g, spos, rows, f);
      precond_store<G>(i, udiag, f, r8, z8, D, dots);
   }
   pdl_trigger();
   store_partials_f<4>(D.red, R_RZ_D, dots, sh);
   if (!last_block(D.state + ST_TICKET0))
      return;
   double tot[4];
   sum_slots_bd(D.red, R_RZ_D, 4, gridDim.x, sh, tot);
   if (threadIdx.x == 0)
      pcg_scalars(tot, D.scal, D.state, D.init, D.n, D.debye, D.poleps, D.politer, D.miniter, D.handle,
         D.use_handle);
}

// ---------------------------------------------------------------------------
// permanent-multipole energy, real space (pair_mpole energy terms,
// include/seq/pair_mpole.h:62-152); exclusion correction (m - 1) x bare pair
// as the reference's exclusion loop does (src/cu/amoeba/empole_cu1.cc:110)

__device__ __forceinline__ float mpole_pair_e(const float* bn, float3 d, const float* mi, const float* mk)
{
   const float dir = mi[1] * d.x + mi[2] * d.y + mi[3] * d.z;
   const float qix = mi[4] * d.x + mi[7] * d.y + mi[8] * d.z;
   const float qiy = mi[7] * d.x + mi[5] * d.y + mi[9] * d.z;
   const float qiz = mi[8] * d.x + mi[9] * d.y + mi[6] * d.z;
   const float qir = qix * d.x + qiy * d.y + qiz * d.z;
   const float dkr = mk[1] * d.x + mk[2] * d.y + mk[3] * d.z;
   const float qkx = mk[4] * d.x + mk[7] * d.y + mk[8] * d.z;
   const float qky = mk[7] * d.x + mk[5] * d.y + mk[9] * d.z;
   const float qkz = mk[8] * d.x + mk[9] * d.y + mk[6] * d.z;
   const float qkr = qkx * d.x + qky * d.y + qkz * d.z;
   const float dik = mi[1] * mk[1] + mi[2] * mk[2] + mi[3] * mk[3];
   const float qik = qix * qkx + qiy * qky + qiz * qkz;
   const float diqk = mi[1] * qkx + mi[2] * qky + mi[3] * qkz;
   const float dkqi = mk[1] * qix + mk[2] * qiy + mk[3] * qiz;
   const float qiqk = 2.f * (mi[7] * mk[7] + mi[8] * mk[8] + mi[9] * mk[9]) + mi[4] * mk[4] + mi[5] * mk[5]
      + mi[6] * mk[6];
   const float t1 = mi[0] * mk[0];
   const float t2 = mk[0] * dir - mi[0] * dkr + dik;
   const float t3 = mi[0] * qkr + mk[0] * qir - dir * dkr + 2.f * (dkqi - diqk + qiqk);
   const float t4 = dir * qkr - dkr * qir - 4.f * qik;
   const float t5 = qir * qkr;
   return t1 * bn[0] + t2 * bn[1] + t3 * bn[2] + t4 * bn[3] + t5 * bn[4];
}

__device__ __forceinline__ void bare_bn5(float f, float invr, float* bn)
{
   const float rr2 = invr * invr;
   bn[0] = f * invr;
   bn[1] = bn[0] * rr2;
   bn[2] = 3.f * bn[1] * rr2;
   bn[3] = 5.f * bn[2] * rr2;
   bn[4] = 7.f * bn[3] * rr2;
}

__device__ __forceinline__ void ewald_bn5(const PairParams& P, float f, float r, float invr, float* bn)
{
   const float rr2 = invr * invr;
   const float ralpha = P.aewald * r;
   const float exp2a = __expf(-ralpha * ralpha);
   float b0 = erfc_hastings(ralpha, exp2a) * invr;
   float b1 = (b0 + P.ec1 * exp2a) * rr2;
   float b2 = (3.f * b1 + P.ec2 * exp2a) * rr2;
   float b3 = (5.f * b2 + P.ec3 * exp2a) * rr2;
   float b4 = (7.f * b3 + P.ec4 * exp2a) * rr2;
   bn[0] = f * b0;
   bn[1] = f * b1;
   bn[2] = f * b2;
   bn[3] = f * b3;
   bn[4] = f * b4;
}

// e_atom[i] = 1/2 sum over i's list and scaled partners (every pair is seen
// from both atoms); FP64 accumulation of FP32 pair energies
template <int G>
__global__ void __launch_bounds__(256) k_empole_real(PairParams P, int npad, float f, ListView nbr,
   const int* __restrict__ nnbr, const int* __restrict__ sp_start, const int* __restrict__ sp_j,
   const float4* __restrict__ sp_sc, const float4* __restrict__ spos, const float* __restrict__ rp,
   double* __restrict__ e_atom)
{
   const int tid = blockIdx.x * blockDim.x + threadIdx.x;
   const int i = tid / G, g = tid % G;
   if (i >= npad)
      return;
   double e = 0;
   if (i < P.n) {
      const float4 pi = spos[i];
      float mi[12];
      load12(rp, i, mi);
      const int cnt = nnbr[i];
      for (int k = g; k < cnt; k += G) {
         const int j = nbr(i, k);
         const float3 d = sep(P, pi, spos[j]);
         const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
         if (r2 <= P.cut2) {
            float mk[12], bn[5];
            load12(rp, j, mk);
            const float invr = rsqrtf(r2);
            if (P.ewald)
               ewald_bn5(P, f, r2 * invr, invr, bn);
            else
               bare_bn5(f, invr, bn);
            e += (double)mpole_pair_e(bn, d, mi, mk);
         }
      }
      const int pa = sp_start[i], pb = sp_start[i + 1];
      for (int q = pa + g; q < pb; q += G) {
         const int j = sp_j[q];
         const float3 d = sep(P, pi, spos[j]);
         const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
         if (r2 <= P.cut2) {
            float mk[12], bn[5];
            load12(rp, j, mk);
            const float invr = rsqrtf(r2);
            const float ms = sp_sc[q].x;
            bare_bn5(f, invr, bn);
            float eb = mpole_pair_e(bn, d, mi, mk);
            if (P.ewald) {
               ewald_bn5(P, f, r2 * invr, invr, bn);
               e += (double)mpole_pair_e(bn, d, mi, mk) + (double)(ms - 1.f) * eb;
            } else {
               e += (double)(ms * eb);
            }
         }
      }
   }
#pragma unroll
   for (int o = G / 2; o > 0; o >>= 1)
      e += __shfl_xor_sync(0xffffffffu, e, o);
   if (g == 0)
      e_atom[i] = i < P.n ? 0.5 * e : 0.0;
}

// ---------------------------------------------------------------------------
// launchers


static constexpr int PAIR_THREADS = 256;

// ---------------------------------------------------------------------------
// Per-step sub-lists, one warp per row.  Each row of the (reused, buffered)
// list is filtered into the pairs within the cutoff and those within the
// preconditioner cutoff, in the row's order (ballot compaction), so the field
// and preconditioner kernels visit only pairs they use, and every entry's
// radial factors are formed here, once per position update: (b1, b2) of the
// mutual field, (b2, b3) of the permanent one and the preconditioner's
// (c1, c2); the same for the scaled partners, by their place in the partner
// table.  Entries within either cutoff queue up in shared memory until a
// warp's worth is there, so the factors (about 130 instructions a pair) are
// formed by full warps although only a quarter to a half of the stored list
// passes.
// STAGE (one CTA per 32-slot block): the block also records which 32-slot
// j-blocks its entries fall in (a bitmap over all blocks in shared memory),
// lists them in ascending order, and rewrites every entry as a local index
// into that list (position x 32 + slot within the j-block), which is where
// the staged kernels find the row in shared memory.
struct FilterOut {
   int lanes_log2;  // of the tiled layout (ListView)
   int cut_cap, pre_cap;  // row capacities
   int* over;       // [LIST_CAPS] largest rows beyond them
   int *nbrc, *nnbrc, *nbrp, *nnbrp;
   float2* cu;  // mutual field
   float2* cd;  // permanent field (b2, b3)
   float2* cp;  // preconditioner
   float2 *spu, *spp;  // scaled partners: mutual field, preconditioner
   int *jbl, *jbn;
   unsigned short *nbrc_l, *nbrp_l;
};

// radial factors of one pair at squared distance r2 and mutual scale us: the
// mutual field's b1, b2 (u), the permanent field's b2, b3 (d; its b1 is the
// mutual one's), the preconditioner's c.  The roundings are written out as
// the kernels that formed the factors in place had them; the two b2 round at
// different points.
__device__ __forceinline__ void pair_factors(const PairParams& P, float r2, float us, float pdi, float pdk,
   float gamma, float polik, float2& u, float2& d, float2& c)
{
   const float invr = rsqrtf(r2);
   const float r = r2 * invr;
   const float rr2 = invr * invr;
   const float rr3 = invr * rr2;
   const float rr5 = 3.f * rr3 * rr2;
   const float rr7 = 5.f * rr5 * rr2;
   float s3, s5, s7;
   thole_damp(r, pdi, gamma, pdk, s3, s5, s7);
   if (P.ewald) {
      const float ralpha = P.aewald * r;
      const float exp2a = __expf(-ralpha * ralpha);
      const float b0 = __fmul_rn(erfc_hastings(ralpha, exp2a), invr);
      const float e1 = __fmul_rn(__fmaf_rn(P.ec1, exp2a, b0), rr2);
      const float y2 = __fmaf_rn(P.ec2, exp2a, __fmul_rn(3.f, e1));
      const float e2 = __fmul_rn(y2, rr2);
      const float y3 = __fmaf_rn(P.ec3, exp2a, __fmul_rn(5.f, e2));
      const float t5 = __fmaf_rn(-us, s5, 1.f);
      u.x = __fmaf_rn(-__fmaf_rn(-us, s3, 1.f), rr3, e1);
      u.y = __fmaf_rn(y2, rr2, -__fmul_rn(t5, rr5));
      d.x = __fmaf_rn(-t5, rr5, e2);
      d.y = __fmaf_rn(-__fmaf_rn(-us, s7, 1.f), rr7, __fmul_rn(y3, rr2));
   } else {
      u.x = us * s3 * rr3;
      u.y = us * s5 * rr5;
      d.x = u.y;
      d.y = us * s7 * rr7;
   }
   const float ir3 = invr * invr * invr;
   c = make_float2(us * s3 * polik * ir3, 3.f * us * s5 * polik * ir3 * invr * invr);
}

// The blocks past the rows' form the scaled partners' factors, a thread per
// entry of the partner table (a warp per row had two lanes at work there).
// PARTS (LIST_...): what to form.  A solve and the fields take everything;
// the energies and forces read the cutoff sub-list alone and the preconditioner
// by itself its own, and would pay for factors that nothing reads (GB300,
// 98,304 atoms, calls after a position update: preconditioner 361 -> 283 us,
// multipole energy without Ewald sum 416 -> 330, van der Waals, which reads
// the stored rows, 580 -> 365; the preconditioner's filter 142 us at five
// blocks an SM, 129 at six, 138 at eight).
template <bool STAGE, int PARTS>
__global__ void __launch_bounds__(STAGE ? 1024 : 256, STAGE ? 1 : PARTS == LIST_PRECOND ? 6 : 5) k_list_filter(PairParams P, float cutp2, int npad,
   const int* __restrict__ nbr, const int* __restrict__ nnbr, const int* __restrict__ sp_j,
   const int* __restrict__ sp_i, int nsp, const float4* __restrict__ sp_sc,
   const float4* __restrict__ spos, const float2* __restrict__ stag, FilterOut O)
{
   extern __shared__ unsigned bits_sm[];
   __shared__ int total_sm;
   constexpr int NW = STAGE ? 32 : 8;
   __shared__ float4 q_d[NW][64];  // separation, partner's pdamp
   __shared__ int q_j[NW][64];
   constexpr bool CUT = PARTS & LIST_CUT, PRE = PARTS & LIST_PRECOND, FIELD = (PARTS & LIST_FIELD) == LIST_FIELD;
   const int blk = blockIdx.x;
   if (blk >= npad / NW) {
      const int q = (blk - npad / NW) * blockDim.x + threadIdx.x;
      if (q >= nsp)
         return;
      const int ii = sp_i[q], js = sp_j[q];
      const float4 pi = spos[ii], pk = spos[js];
      const float2 ti = stag[ii], tk = stag[js];
      const float3 d = sep(P, pi, pk);
      const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
      float2 u, f, c;
      pair_factors(P, r2, sp_sc[q].w, pi.w, pk.w, pair_gamma(P, ti.x, tk.x), ti.y * tk.y, u, f, c);
      // zero factors beyond the cutoff
      if (FIELD)
         O.spu[q] = r2 <= P.cut2 ? u : make_float2(0.f, 0.f);
      if (PRE)
         O.spp[q] = r2 <= cutp2 ? c : make_float2(0.f, 0.f);
      return;
   }
   const int words = (npad / 32 + 31) / 32;
   unsigned* bm = bits_sm;
   int* pre = reinterpret_cast<int*>(bits_sm + words);
   if (STAGE) {
      for (int w = threadIdx.x; w < words; w += blockDim.x)
         bm[w] = 0u;
      __syncthreads();
   }
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int i = blk * NW + warp;
   const ListView VC{nullptr, O.cut_cap, O.lanes_log2}, VP{nullptr, O.pre_cap, O.lanes_log2};
   int oc = 0, op = 0;
   if (i < P.n) {
      const float4 pi = spos[i];
      const float2 ti = stag[i];  // thole or type, polarizability
      const int* row = nbr + (size_t)i * P.cap;
      const int cnt = nnbr[i];
      const float rmax2 = CUT && PRE ? fmaxf(P.cut2, cutp2) : CUT ? P.cut2 : cutp2;
      const unsigned lt = (1u << lane) - 1u;
      // the row's place in the tiled lists, and an entry's from it
      const size_t base = VC.at(i, 0), basep = VP.at(i, 0);
      int* nc = O.nbrc + base;
      float2* cu = O.cu + base;
      float2* cd = O.cd + base;
      int* np = O.nbrp + basep;
      float2* cp = O.cp + basep;
      const int sg = O.lanes_log2, gm = (1 << sg) - 1;
      int qn = 0;
      // the first m (<= 32) queued entries into the sub-lists
      const auto drain = [&](int m) {
         const bool valid = lane < m;
         const int j = valid ? q_j[warp][lane] : i;
         const float2 tk = stag[j];
         const float4 dk = valid ? q_d[warp][lane] : make_float4(1.f, 0.f, 0.f, 1.f);
         const float r2 = dk.x * dk.x + dk.y * dk.y + dk.z * dk.z;
         const bool inc = CUT && valid && r2 <= P.cut2, inp = PRE && valid && r2 <= cutp2;
         const unsigned mc = __ballot_sync(0xffffffffu, inc), mp = __ballot_sync(0xffffffffu, inp);
         float2 u, f, c;
         pair_factors(P, r2, 1.f, pi.w, dk.w, pair_gamma(P, ti.x, tk.x), ti.y * tk.y, u, f, c);
         if (inc) {
            const unsigned k = oc + __popc(mc & lt), at = ((k >> sg) << 5) + (k & gm);
            if (k < (unsigned)O.cut_cap) {
               nc[at] = j;
               if (FIELD) {
                  cu[at] = u;
                  cd[at] = f;
               }
            }
         }
         if (inp) {
            const unsigned k = op + __popc(mp & lt), at = ((k >> sg) << 5) + (k & gm);
            if (k < (unsigned)O.pre_cap) {
               np[at] = j;
               cp[at] = c;
            }
         }
         if (STAGE && (inc || inp))
            atomicOr(&bm[j >> 10], 1u << ((j >> 5) & 31));
         oc += __popc(mc);
         op += __popc(mp);
      };
      int j = lane < cnt ? row[lane] : i;
      for (int k0 = 0; k0 < cnt; k0 += 32) {
         const bool in = k0 + lane < cnt;
         const float4 pk = spos[j];
         const int jn = k0 + 32 + lane < cnt ? row[k0 + 32 + lane] : i;
         const float3 d = sep(P, pi, pk);
         const bool acc = in && d.x * d.x + d.y * d.y + d.z * d.z <= rmax2;
         const unsigned m = __ballot_sync(0xffffffffu, acc);
         if (PARTS == LIST_CUT) {  // indices alone: nothing to queue for
            const unsigned k = oc + __popc(m & lt);
            if (acc && k < (unsigned)O.cut_cap)
               nc[((k >> sg) << 5) + (k & gm)] = j;
            oc += __popc(m);
            j = jn;
            continue;
         }
         if (acc) {
            const int p = qn + __popc(m & lt);
            q_d[warp][p] = make_float4(d.x, d.y, d.z, pk.w);
            q_j[warp][p] = j;
         }
         qn += __popc(m);
         j = jn;
         __syncwarp();
         if (qn >= 32) {
            drain(32);
            qn -= 32;
            __syncwarp();
            if (lane < qn) {
               q_d[warp][lane] = q_d[warp][32 + lane];
               q_j[warp][lane] = q_j[warp][32 + lane];
            }
            __syncwarp();
         }
      }
      if (qn > 0)
         drain(qn);
   }
   if (lane == 0 && CUT && oc > O.cut_cap)
      atomicMax(O.over + 1, oc);
   if (lane == 0 && PRE && op > O.pre_cap)
      atomicMax(O.over + 2, op);
   oc = min(oc, O.cut_cap);
   op = min(op, O.pre_cap);
   if (lane == 0) {
      if (CUT)
         O.nnbrc[i] = oc;
      if (PRE)
         O.nnbrp[i] = op;
   }
   if (!STAGE)
      return;
   __syncthreads();
   // set bits before each word, and the block's j-block list
   if (warp == 0) {
      int run = 0;
      for (int w0 = 0; w0 < words; w0 += 32) {
         const int w = w0 + lane;
         const int c = w < words ? __popc(bm[w]) : 0;
         int incl = c;
#pragma unroll
         for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
               incl += t;
         }
         if (w < words)
            pre[w] = run + incl - c;
         run += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) {
         total_sm = run;
         O.jbn[blk] = run;
      }
   }
   __syncthreads();
   const int total = total_sm;
   if (total > STAGE_JB_CAP)
      return;  // this block reads its rows from global memory
   for (int w = threadIdx.x; w < words; w += blockDim.x) {
      unsigned m = bm[w];
      int q = pre[w];
      while (m) {
         const int b = __ffs(m) - 1;
         O.jbl[(size_t)blk * STAGE_JB_CAP + q] = w * 32 + b;
         ++q;
         m &= m - 1u;
      }
   }
   if (i < P.n) {
      unsigned short* lc = O.nbrc_l + (size_t)i * O.cut_cap;
      unsigned short* lp = O.nbrp_l + (size_t)i * O.pre_cap;
      for (int k = lane; k < oc; k += 32) {
         const int j = O.nbrc[VC.at(i, k)], jb = j >> 5;
         const int q = pre[jb >> 5] + __popc(bm[jb >> 5] & ((1u << (jb & 31)) - 1u));
         lc[k] = (unsigned short)(q * 32 + (j & 31));
      }
      for (int k = lane; k < op; k += 32) {
         const int j = O.nbrp[VP.at(i, k)], jb = j >> 5;
         const int q = pre[jb >> 5] + __popc(bm[jb >> 5] & ((1u << (jb & 31)) - 1u));
         lp[k] = (unsigned short)(q * 32 + (j & 31));
      }
   }
}

int launch_list_filter(Context* ctx, int parts)
{
   const bool cut = parts == LIST_CUT && !ctx->pair_staged, pre = parts == LIST_PRECOND && !ctx->pair_staged;
   PairParams P = make_params(ctx, ctx->cfg.cutoff);
   const double cp = ctx->cfg.usolve_cutoff + ctx->cfg.pbuffer;
   const float cutp2 = cp * cp > 3.0e38 ? 3.0e38f : (float)(cp * cp);
   const int nblk = ctx->npad / 32;
   const int words = (nblk + 31) / 32;
   const size_t smem = sizeof(unsigned) * 2 * (size_t)words;
   const int* nbr = ctx->nbre ? ctx->nbre : ctx->nbr;
   const int* nnbr = ctx->nbre ? ctx->nnbre : ctx->nnbr;
   ctx->list_lanes = ctx->pair_lanes;
   FilterOut O{nbrc_view(ctx).sg, ctx->cut_cap, ctx->pre_cap, ctx->nbr_over, ctx->nbrc, ctx->nnbrc, ctx->nbrp, ctx->nnbrp, ctx->cfu, ctx->cfd, ctx->cfp, ctx->spu,
      ctx->spp, ctx->jbl, ctx->jbn, ctx->nbrc_l, ctx->nbrp_l};
   if (ctx->pair_staged)
      k_list_filter<true, LIST_ALL><<<nblk + grid_for(ctx->nsp, 1024), 1024, smem, ctx->stream>>>(P, cutp2, ctx->npad,
         nbr, nnbr, ctx->sp_j, ctx->sp_i, ctx->nsp, ctx->sp_sc, ctx->spos, ctx->stag, O);
   else {
      auto k = cut ? k_list_filter<false, LIST_CUT> : pre ? k_list_filter<false, LIST_PRECOND>
                                                          : k_list_filter<false, LIST_ALL>;
      k<<<ctx->npad / 8 + (cut ? 0 : grid_for(ctx->nsp, 256)), 256, 0, ctx->stream>>>(P, cutp2, ctx->npad, nbr,
         nnbr, ctx->sp_j, ctx->sp_i, ctx->nsp, ctx->sp_sc, ctx->spos, ctx->stag, O);
   }
   ctx->list_have = cut || pre ? parts : LIST_ALL;
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

// Where the grid leaves an SM at most one block, a row's trips wait on their
// own latency, not on the L1's line rate: four entries a trip (80-106
// registers).  GB300, a solve from alpha E: droplets of 648 / 1,500 / 2,100 atoms
// (rows of all atoms) 319 / 702 / 1,212 -> 297 / 623 / 863 us; periodic boxes of
// 648 to 3,072 atoms the same either way; at 12,288 atoms two entries are better
// (670 against 722).
static bool few_blocks(int nb) { return nb <= 152; }

static TensorList field_list(const Context* ctx) { return {ctx->nbrc, ctx->nnbrc, ctx->cfu, ctx->spu}; }
static TensorList precond_list(const Context* ctx) { return {ctx->nbrp, ctx->nnbrp, ctx->cfp, ctx->spp}; }
static Partners partners(const Context* ctx) { return {ctx->sp_start, ctx->sp_j}; }

// lanes per atom of the three field kernels (4, 8, 16 or 32; t9gb_pair_lanes)
#define T9_LANES_DISPATCH(KERNEL, ...)                                                                                 \
   do {                                                                                                                \
      const int g_ = ctx->pair_lanes;                                                                                  \
      const int nb_ = grid_for((long long)ctx->npad * g_, PAIR_THREADS);                                               \
      if (g_ == 4)                                                                                                     \
         KERNEL<4><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                                \
      else if (g_ == 8)                                                                                                \
         KERNEL<8><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                                \
      else if (g_ == 32)                                                                                               \
         KERNEL<32><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                               \
      else                                                                                                             \
         KERNEL<16><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                               \
   } while (0)

// the same for kernels with a second template parameter
#define T9_LANES_DISPATCH2(KERNEL, ARG, ...)                                                                           \
   do {                                                                                                                \
      const int g_ = ctx->pair_lanes;                                                                                  \
      const int nb_ = grid_for((long long)ctx->npad * g_, PAIR_THREADS);                                               \
      if (g_ == 4)                                                                                                     \
         KERNEL<4, ARG><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                           \
      else if (g_ == 8)                                                                                                \
         KERNEL<8, ARG><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                           \
      else if (g_ == 32)                                                                                               \
         KERNEL<32, ARG><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                          \
      else                                                                                                             \
         KERNEL<16, ARG><<<nb_, PAIR_THREADS, 0, ctx->stream>>>(__VA_ARGS__);                                          \
   } while (0)

// the staged kernels: 4 or 8 lanes per atom
static bool staged_lanes(const Context* ctx)
{
   return ctx->pair_staged && (ctx->pair_lanes == 4 || ctx->pair_lanes == 8);
}

int pair_staging_setup()
{
   const int bytes = (int)STAGE_SMEM;
   if (cudaFuncSetAttribute(k_ufield_stg<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||
      cudaFuncSetAttribute(k_ufield_stg<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||
      cudaFuncSetAttribute(k_precond_dots_stg<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
         cudaSuccess ||
      cudaFuncSetAttribute(k_precond_dots_stg<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
      return T9GB_CUDA_ERR;
   // the block bitmap and its prefix counts: 8 bytes per 1,024 slots
   if (cudaFuncSetAttribute(k_list_filter<true, LIST_ALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024) !=
      cudaSuccess)
      return T9GB_CUDA_ERR;
   return T9GB_OK;
}

// parameters of the kernels over the two sub-lists (cap: their row capacity)
static PairParams field_params(const Context* ctx)
{
   PairParams P = make_params(ctx, ctx->cfg.cutoff);
   P.cap = ctx->cut_cap;
   return P;
}

static PairParams precond_params(const Context* ctx)
{
   PairParams P = make_params(ctx, ctx->cfg.usolve_cutoff + ctx->cfg.pbuffer);
   P.ewald = 0;
   P.cap = ctx->pre_cap;
   return P;
}

int launch_ufield_real(Context* ctx, const float* u6, const float* base6, float* out6)
{
   PairParams P = field_params(ctx);
   prof_begin(ctx, P_UFIELD_REAL);
   if (staged_lanes(ctx)) {
      auto k = ctx->pair_lanes == 8 ? k_ufield_stg<8> : k_ufield_stg<4>;
      T9_CUDA(launch_k(use_pdl(ctx), k, ctx->npad / 32, 32 * ctx->pair_lanes, STAGE_SMEM, ctx->stream, P,
         field_list(ctx), partners(ctx), ctx->nbrc_l, ctx->jbl, ctx->jbn, ctx->spos, u6, base6, out6, ctx->copy_err));
      prof_end(ctx);
      return T9GB_OK;
   }
   const int g = ctx->pair_lanes;
   const int nb = grid_for((long long)ctx->npad * g, PAIR_THREADS);
   auto k = g == 4 ? k_ufield_real<4, false> : g == 8 ? k_ufield_real<8, false> : g == 32 ? k_ufield_real<32, false>
                                                                                    : k_ufield_real<16, false>;
   if (g == 8 && few_blocks(nb))
      k = k_ufield_real<8, false, 4>;
   else if (g == 16 && few_blocks(nb))
      k = k_ufield_real<16, false, 4>;
   T9_CUDA(launch_k(use_pdl(ctx), k, nb, PAIR_THREADS, 0, ctx->stream, P, ctx->npad, field_list(ctx),
      partners(ctx), ctx->spos, u6, nullptr, nullptr, base6, out6));
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_ufield_real_dir(Context* ctx, const float* p6, const float* z6, const double* scal, float* out6)
{
   PairParams P = field_params(ctx);
   prof_begin(ctx, P_UFIELD_REAL);
   T9_LANES_DISPATCH2(k_ufield_real, true, P, ctx->npad, field_list(ctx), partners(ctx), ctx->spos, p6, z6, scal,
      nullptr, out6);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_dfield_real(Context* ctx, const float* base6, float* out6)
{
   PairParams P = field_params(ctx);
   prof_begin(ctx, P_DFIELD_REAL);
   T9_LANES_DISPATCH(k_dfield_real, P, ctx->npad, field_list(ctx), ctx->cfd, ctx->sp_start, ctx->sp_j, ctx->sp_sc, ctx->spos,
      ctx->srpole, base6, ctx->exfld, out6);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_precond_sparse_dots(Context* ctx, const float* r6, float* z6, const PcgDots& D)
{
   PairParams P = precond_params(ctx);
   const int g = ctx->pair_lanes;
   const int per = PAIR_THREADS / g;
   const int nb = std::min(RED_MAX, (ctx->npad + per - 1) / per);
   prof_begin(ctx, P_PRECOND);
   if (staged_lanes(ctx)) {
      const int nblk = ctx->npad / 32;
      auto ks = g == 8 ? k_precond_dots_stg<8> : k_precond_dots_stg<4>;
      T9_CUDA(launch_k(use_pdl(ctx), ks, std::min(RED_MAX, nblk), 32 * g, STAGE_SMEM, ctx->stream, P, nblk,
         (float)ctx->cfg.udiag, precond_list(ctx), partners(ctx), ctx->nbrp_l, ctx->jbl, ctx->jbn, ctx->spos, r6, z6, D,
         ctx->copy_err));
      prof_end(ctx);
      return T9GB_OK;
   }
   auto k = g == 4 ? k_precond_sparse_dots<4> : g == 8 ? k_precond_sparse_dots<8> : g == 32
         ? k_precond_sparse_dots<32> : k_precond_sparse_dots<16>;
   if (g == 8 && few_blocks(nb))
      k = k_precond_sparse_dots<8, 4>;
   else if (g == 16 && few_blocks(nb))
      k = k_precond_sparse_dots<16, 4>;
   T9_CUDA(launch_k(use_pdl(ctx), k, nb, PAIR_THREADS, 0, ctx->stream, P, ctx->npad, (float)ctx->cfg.udiag, precond_list(ctx),
      partners(ctx), ctx->spos, r6, z6, D));
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

int launch_precond_sparse(Context* ctx, const float* r6, float* z6)
{
   PairParams P = precond_params(ctx);
   prof_begin(ctx, P_PRECOND);
   T9_LANES_DISPATCH(k_precond_sparse, P, ctx->npad, (float)ctx->cfg.udiag, precond_list(ctx), partners(ctx),
      ctx->spos, r6, z6);
   prof_end(ctx);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}

}  // namespace t9gb

namespace t9gb {
int launch_empole_real(Context* ctx, double* e_atom)
{
   PairParams P = make_params(ctx, ctx->cfg.cutoff);
   k_empole_real<GROUP><<<grid_for((long long)ctx->npad * GROUP, PAIR_THREADS), PAIR_THREADS, 0, ctx->stream>>>(P,
      ctx->npad, (float)ctx->cfg.electric, nbrc_view(ctx), ctx->nnbrc, ctx->sp_start, ctx->sp_j, ctx->sp_sc, ctx->spos,
      ctx->srpole, e_atom);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}
}  // namespace t9gb

// ---------------------------------------------------------------------------
// Descriptors of the learned initial guess.  Per slot i two rows of 32
// features, row i for the d dipoles and row npad + i for the p dipoles; every
// vector is expressed in the atom's local multipole frame (rows of
// sframe[9]), so the features are invariant under rotations of the system:
//   0-2   direct field E (d or p)
//   3     polarizability alpha_i
//   4-10  sum_k fc(r) g(r; mu, 0.5), mu = 1, 1.83, ..., 6            (count)
//   11-14 sum_k q_k fc g(r; mu, 0.75), mu = 1.5, 3, 4.5, 6           (charge)
//   15-20 sum_k q_k fc g(r; mu, 1) r_hat, mu = 2, 4.5 (x, y, z each)  (charge
//         direction)
//   21-25 sum_k alpha_k fc g(r; mu, 0.6), mu = 1, 2.25, ..., 6     (polarizability)
//   26-31 first-order mutual field of the neighbours' direct dipoles,
//         sum_k -T_ik^Thole (alpha_k E_k) * u-scale, split r < 3.5 / r >= 3.5
// over all partners within 6 A; fc = (1 + cos(pi r / 6)) / 2.
// g(r; mu, s) = exp(-(r - mu)^2 / (2 s^2)).

namespace t9gb {

constexpr float DESC_CUT = 6.f;
constexpr int NFEAT = 32;

__device__ __forceinline__ float gauss(float r, float mu, float inv2s2)
{
   const float t = r - mu;
   return __expf(-t * t * inv2s2);
}

// acc[j] += w g(r; mu0 + j dmu, s), j < N, c = 1 / (2 s^2), by the product
// recurrence g_{j+1} = g_j R_j, R_j = exp(c (2 dmu (r - mu0) - dmu^2))
// exp(-2 c dmu^2)^j: two exponentials per series instead of N (relative
// error a few units of 1e-7 over the series)
template <int N>
__device__ __forceinline__ void gauss_series(float r, float mu0, float dmu, float c, float w, float* acc)
{
   const float t = r - mu0;
   float g = __expf(-t * t * c);
   float R = __expf(c * (2.f * dmu * t - dmu * dmu));
   const float B = __expf(-2.f * c * dmu * dmu);  // constant: folded by the compiler
#pragma unroll
   for (int j = 0; j < N; ++j) {
      acc[j] += w * g;
      g *= R;
      R *= B;
   }
}

// acc layout: gr[0..7) gq[7..11) dq[11..17) ga[17..22) fd[22..28) fp[28..34)
constexpr int DACC = 34;

__device__ __forceinline__ void desc_pair(const PairParams& P, float r2, float3 d, float us, float pdi, float pti, float pdk,
   const float* uk, float qk, float* acc)
{
   const float invr = rsqrtf(r2);
   const float r = r2 * invr;
   const float fc = 0.5f * (__cosf(3.14159265f / DESC_CUT * r) + 1.f);
   gauss_series<7>(r, 1.f, 5.f / 6.f, 2.f, fc, acc);
   gauss_series<4>(r, 1.5f, 1.5f, 1.f / (2.f * 0.75f * 0.75f), qk * fc, acc + 7);
   const float h0 = qk * fc * gauss(r, 2.f, 0.5f) * invr, h1 = qk * fc * gauss(r, 4.5f, 0.5f) * invr;
   acc[11] += h0 * d.x;
   acc[12] += h0 * d.y;
   acc[13] += h0 * d.z;
   acc[14] += h1 * d.x;
   acc[15] += h1 * d.y;
   acc[16] += h1 * d.z;
   gauss_series<5>(r, 1.f, 1.25f, 1.f / (2.f * 0.6f * 0.6f), uk[7] * fc, acc + 17);
   float s3, s5, s7;
   thole_damp(r, pdi, pair_gamma(P, pti, uk[6]), pdk, s3, s5, s7);
   const float ir3 = invr * invr * invr;
   const float rr3 = us * s3 * ir3;
   const float rr5 = 3.f * us * s5 * ir3 * invr * invr;
   const float cd = rr5 * (d.x * uk[0] + d.y * uk[1] + d.z * uk[2]);
   const float cp = rr5 * (d.x * uk[3] + d.y * uk[4] + d.z * uk[5]);
   // constant indices in both branches keep acc in registers
   if (r < 3.5f) {
      acc[22] += cd * d.x - rr3 * uk[0];
      acc[23] += cd * d.y - rr3 * uk[1];
      acc[24] += cd * d.z - rr3 * uk[2];
      acc[28] += cp * d.x - rr3 * uk[3];
      acc[29] += cp * d.y - rr3 * uk[4];
      acc[30] += cp * d.z - rr3 * uk[5];
   } else {
      acc[25] += cd * d.x - rr3 * uk[0];
      acc[26] += cd * d.y - rr3 * uk[1];
      acc[27] += cd * d.z - rr3 * uk[2];
      acc[31] += cp * d.x - rr3 * uk[3];
      acc[32] += cp * d.y - rr3 * uk[4];
      acc[33] += cp * d.z - rr3 * uk[5];
   }
}

__device__ __forceinline__ void to_local(const float* F, const float* v, float* out)
{
#pragma unroll
   for (int a = 0; a < 3; ++a)
      out[a] = F[3 * a] * v[0] + F[3 * a + 1] * v[1] + F[3 * a + 2] * v[2];
}

template <int G>
__global__ void __launch_bounds__(256) k_learn_features(PairParams P, int npad, ListView nbr,
   const int* __restrict__ nnbr, const int* __restrict__ sp_start, const int* __restrict__ sp_j,
   const float4* __restrict__ sp_sc, const float4* __restrict__ spos, const float* __restrict__ srpole,
   const float* __restrict__ sframe, const float* __restrict__ e8, const float* __restrict__ u8,
   float* __restrict__ xf, const float* __restrict__ polar, const float* __restrict__ fstat,
   const int* __restrict__ state, __nv_bfloat16* __restrict__ xn)
{
   const int tid = blockIdx.x * blockDim.x + threadIdx.x;
   const int i = tid / G, g = tid % G;
   if (i >= npad)
      return;
   // with the column statistics fixed (bit 0), also the BF16 network input
   const bool norm = (state[ST_LREADY] & 1) != 0;
   float acc[DACC];
#pragma unroll
   for (int c = 0; c < DACC; ++c)
      acc[c] = 0.f;
   if (i < P.n) {
      const float4 pi = spos[i];
      const float pti = u8[8 * i + 6];
      const int cnt = nnbr[i];
      for (int k = g; k < cnt; k += G) {
         const int j = nbr(i, k);
         const float4 pk = spos[j];
         const float3 d = sep(P, pi, pk);
         const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
         if (r2 < DESC_CUT * DESC_CUT) {
            float uk[8];
            load8(u8, j, uk);
            desc_pair(P, r2, d, 1.f, pi.w, pti, pk.w, uk, srpole[12 * j], acc);
         }
      }
      const int pa = sp_start[i], pb = sp_start[i + 1];
      for (int q = pa + g; q < pb; q += G) {
         const int j = sp_j[q];
         const float4 pk = spos[j];
         const float3 d = sep(P, pi, pk);
         const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
         if (r2 < DESC_CUT * DESC_CUT) {
            float uk[8];
            load8(u8, j, uk);
            desc_pair(P, r2, d, sp_sc[q].w, pi.w, pti, pk.w, uk, srpole[12 * j], acc);
         }
      }
   }
   group_reduce<G, DACC>(acc);
   if (g >= 2)
      return;
   // lane 0 writes the d row, lane 1 the p row
   const size_t row = (size_t)(g == 0 ? i : npad + i);
   float x[NFEAT];
#pragma unroll
   for (int c = 0; c < NFEAT; ++c)
      x[c] = 0.f;
   if (i < P.n) {
      float F[9];
#pragma unroll
      for (int c = 0; c < 9; ++c)
         F[c] = sframe[9 * i + c];
      float v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
         v[c] = e8[8 * i + 3 * g + c];
      to_local(F, v, x);
      x[3] = u8[8 * i + 7];
#pragma unroll
      for (int c = 0; c < 7; ++c)
         x[4 + c] = acc[c];
#pragma unroll
      for (int c = 0; c < 4; ++c)
         x[11 + c] = acc[7 + c];
      to_local(F, acc + 11, x + 15);
      to_local(F, acc + 14, x + 18);
#pragma unroll
      for (int c = 0; c < 5; ++c)
         x[21 + c] = acc[17 + c];
      float f[6];
#pragma unroll
      for (int c = 0; c < 6; ++c)
         f[c] = g == 0 ? acc[22 + c] : acc[28 + c];
      to_local(F, f, x + 26);
      to_local(F, f + 3, x + 29);
   }
   float4* xo = reinterpret_cast<float4*>(xf + row * NFEAT);
#pragma unroll
   for (int c = 0; c < NFEAT; c += 4)
      xo[c / 4] = make_float4(x[c], x[c + 1], x[c + 2], x[c + 3]);
   if (norm) {  // as k_normalize: (x - mean) / std, zero rows where alpha = 0
      const bool live = polar[i] != 0.f;
      uint4* q = reinterpret_cast<uint4*>(xn + row * NFEAT);
#pragma unroll
      for (int c = 0; c < NFEAT; c += 8) {
         unsigned wv[4];
#pragma unroll
         for (int k = 0; k < 4; ++k) {
            const int a = c + 2 * k;
            const float v0 = live ? (x[a] - fstat[a]) * fstat[32 + a] : 0.f;
            const float v1 = live ? (x[a + 1] - fstat[a + 1]) * fstat[32 + a + 1] : 0.f;
            const __nv_bfloat162 b = __floats2bfloat162_rn(v0, v1);
            wv[k] = *reinterpret_cast<const unsigned*>(&b);
         }
         q[c / 8] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
      }
   }
}

int launch_learn_features(Context* ctx, const float* e8, const float* u8, float* xf, const float* fstat,
   __nv_bfloat16* xn)
{
   PairParams P = make_params(ctx, DESC_CUT);
   k_learn_features<GROUP><<<grid_for((long long)ctx->npad * GROUP, PAIR_THREADS), PAIR_THREADS, 0, ctx->stream>>>(P,
      ctx->npad, ctx->cfg.cutoff >= DESC_CUT ? nbrc_view(ctx) : nbr_view(ctx), ctx->cfg.cutoff >= DESC_CUT ? ctx->nnbrc : ctx->nnbr,
      ctx->sp_start, ctx->sp_j, ctx->sp_sc, ctx->spos, ctx->srpole, ctx->sframe, e8, u8, xf, ctx->spolar, fstat,
      ctx->status, xn);
   T9_CUDA(cudaGetLastError());
   return T9GB_OK;
}
}  // namespace t9gb
