// Allocation-free variant of the mutual-field kernel (t9gb_ufield_noalloc).
//
// Some callers cannot call cudaMalloc at the point where they need the
// field: host programs that own every device allocation themselves (a
// plugin must not grow the footprint behind the host's allocator), code that
// runs while a stream is being captured into a CUDA graph (an allocation
// would break the capture), and real-time loops that forbid allocator calls
// after start-up.  This entry point serves them: the caller passes device
// inputs and outputs, and a call takes one launch and no working memory
// (where an output overlaps an input, the inputs are first copied to a fixed
// array in the library's own device image).
//
// Scope: the damped (non-Ewald) mutual field -T u for d and p dipoles within
// a cutoff, minimum image in an orthorhombic box or no box, every pair with
// mutual scale 1 (the AMOEBA mutual-11..14 scales; the reference's CUDA
// ufield also runs with an empty uexclude table).  All pairs are visited, so
// the size is capped at T9GB_NOALLOC_MAX_ATOMS.
#include <mutex>

#include "common.cuh"
#include "reduce.cuh"

namespace t9gb {

constexpr int NA_WARPS = 8;     // atoms per block, one a warp
constexpr int NA_STEP = 2;      // groups of 32 partners tested at a time
constexpr int NA_CHUNK = 1024;  // positions staged at a time: a group for each lane
constexpr int NA_QUEUE = 64;    // queued pairs per atom, a ring

// Working memory of a call whose outputs overlap its inputs: the inputs are
// copied here first.  Every GPU that loads the library keeps this array
// (352 KiB) until the process exits.
static __device__ __align__(256) float g_noalloc_scratch[11 * T9GB_NOALLOC_MAX_ATOMS];

// Device address of the array, looked up once per device.
static std::mutex g_noalloc_mu;
static float* g_noalloc_ptr[64] = {nullptr};

static int noalloc_scratch(int dev, float** out)
{
   std::lock_guard<std::mutex> lock(g_noalloc_mu);
   if (!g_noalloc_ptr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p)
         return T9GB_CUDA_ERR;
      g_noalloc_ptr[dev] = static_cast<float*>(p);
   }
   *out = g_noalloc_ptr[dev];
   return T9GB_OK;
}

__global__ void k_noalloc_copy(int n, const float* __restrict__ xyz, const float* __restrict__ pdamp,
   const float* __restrict__ thole, const float* __restrict__ uind, const float* __restrict__ uinp,
   float* __restrict__ to)
{
   const int k = blockIdx.x * blockDim.x + threadIdx.x;
   if (k >= 3 * n)
      return;
   to[k] = xyz[k];
   to[3 * n + k] = uind[k];
   to[6 * n + k] = uinp[k];
   if (k < n) {
      to[9 * n + k] = pdamp[k];
      to[10 * n + k] = thole[k];
   }
}

// d - l rint(d linv), bit for bit for |d linv| < 2^22: the sum with 1.5 2^23
// rounds to an integer on the FP32 pipe, where rint has a pipe of an eighth
// of the rate (beyond 2^22 box lengths an FP32 position does not resolve the
// box)
__device__ __forceinline__ float na_image(float d, float l, float linv)
{
   const float big = 12582912.f, k = __fadd_rn(__fmul_rn(d, linv), big);
   return d - l * __fsub_rn(k, big);
}

// one queued pair (dx, dy, dz, j) seen from i
__device__ __forceinline__ void na_pair(float4 p, int i, float pdi, float pti, const float* __restrict__ pdamp,
   const float* __restrict__ thole, const float* __restrict__ uind, const float* __restrict__ uinp, float* f)
{
   const int j = __float_as_int(p.w);
   if (j == i)
      return;
   const float dx = p.x, dy = p.y, dz = p.z;
   const float udx = uind[3 * j], udy = uind[3 * j + 1], udz = uind[3 * j + 2];
   const float upx = uinp[3 * j], upy = uinp[3 * j + 1], upz = uinp[3 * j + 2];
   const float r2 = dx * dx + dy * dy + dz * dz;
   const float invr = rsqrtf(r2);
   const float r = r2 * invr;
   // Thole damping (include/seq/damp.h:8-24) and the damped tensor
   // (include/seq/pair_field.h:333-420, non-Ewald branch, u-scale 1)
   const float pgamma = fminf(pti, thole[j]);
   float damp = pdi * pdamp[j];
   const float ratio = r * __frcp_rn(damp);
   damp = (damp == 0.f) ? -1.0e16f : -pgamma * ratio * ratio * ratio;
   const float ex = __expf(damp);
   const float rr3 = invr * invr * invr;
   const float b1 = (1.f - ex) * rr3;
   const float b2 = (1.f - ex * (1.f - damp)) * 3.f * rr3 * invr * invr;
   float c = b2 * (dx * udx + dy * udy + dz * udz);
   f[0] += c * dx - b1 * udx;
   f[1] += c * dy - b1 * udy;
   f[2] += c * dz - b1 * udz;
   c = b2 * (dx * upx + dy * upy + dz * upz);
   f[3] += c * dx - b1 * upx;
   f[4] += c * dy - b1 * upy;
   f[5] += c * dz - b1 * upz;
}

// floats as integers of the same order
__device__ __forceinline__ int na_key(float x)
{
   const int b = __float_as_int(x);
   return b ^ (b >> 31 & 0x7fffffff);
}
__device__ __forceinline__ float na_unkey(int k) { return __int_as_float(k ^ (k >> 31 & 0x7fffffff)); }

// One warp per atom i.  The block stages the positions, and the bounding box
// of each 32 of them; a lane tests one box against i, and the warp tests the
// atoms of the boxes within reach, NA_STEP boxes at a time.  The pairs within
// the cutoff go to a ring, and a full warp of them is evaluated at once.
//
// What bounds it: a small call is one launch (the inputs are read where they
// are; with 16 lanes an atom over packed records it took two: 8.2 -> 5.2 us a
// call at 648 atoms), a large one the issue of the n^2 distance tests, about
// 30 instructions for 32 pairs.  Boxes drop the groups out of reach (half to
// nine tenths of a box whose atoms are in the order of their molecules; in a
// random order the boxes cost a tenth), and the queue keeps the pair term off
// the tests, of which 2 % hit at 7,500 atoms.  In a stream, 1,536 / 4,000 /
// 7,500 atoms at a cutoff of 7: 39 / 84 / 143 -> 11 / 23 / 51 us; without the
// boxes 12 / 30 / 79.  Blocks of 4 and 16 warps take 70 and 48 us at 7,500
// and 10.0 and 9.2 instead of 8.2 us at 648.
__global__ void __launch_bounds__(32 * NA_WARPS) k_noalloc_ufield(int n, float lx, float ly, float lz, float ilx,
   float ily, float ilz, float cut2, const float* __restrict__ xyz, const float* __restrict__ pdamp,
   const float* __restrict__ thole, const float* __restrict__ uind, const float* __restrict__ uinp,
   float* __restrict__ field, float* __restrict__ fieldp)
{
   __shared__ float sx[3 * NA_CHUNK];
   __shared__ float box[6][NA_CHUNK / 32];
   __shared__ float4 ring[NA_WARPS][NA_QUEUE];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const unsigned lt = (1u << lane) - 1;
   const int i = blockIdx.x * NA_WARPS + w, ic = min(i, n - 1);
   const float px = xyz[3 * ic], py = xyz[3 * ic + 1], pz = xyz[3 * ic + 2];
   const float pdi = pdamp[ic], pti = thole[ic];
   float f[6] = {0, 0, 0, 0, 0, 0};
   int head = 0, tail = 0;
   for (int c0 = 0; c0 < n; c0 += NA_CHUNK) {
      const int m = min(NA_CHUNK, n - c0), groups = (m + 31) / 32;
      __syncthreads();
      for (int k = threadIdx.x; k < 3 * m; k += 32 * NA_WARPS)
         sx[k] = xyz[3 * c0 + k];
      __syncthreads();
      for (int q = w; q < groups; q += NA_WARPS) {
         const int jl = min(32 * q + lane, m - 1);
         float lo[3], hi[3];
#pragma unroll
         for (int c = 0; c < 3; ++c) {
            const int key = na_key(sx[3 * jl + c]);
            lo[c] = na_unkey(__reduce_min_sync(0xffffffffu, key));
            hi[c] = na_unkey(__reduce_max_sync(0xffffffffu, key));
         }
         if (lane < 3) {
            const float l = lane == 0 ? lo[0] : (lane == 1 ? lo[1] : lo[2]);
            const float h = lane == 0 ? hi[0] : (lane == 1 ? hi[1] : hi[2]);
            box[lane][q] = 0.5f * (l + h);
            box[3 + lane][q] = 0.5f * (h - l);
         }
      }
      __syncthreads();
      // the boxes within reach of i; the slack covers the roundings of the
      // box, of the image and of the distance
      bool near = i < n && lane < groups;
      if (near) {
         float r2 = 0.f;
#pragma unroll
         for (int c = 0; c < 3; ++c) {
            const float p = c == 0 ? px : (c == 1 ? py : pz), l = c == 0 ? lx : (c == 1 ? ly : lz);
            const float m0 = box[c][lane];
            const float d = fabsf(na_image(m0 - p, l, c == 0 ? ilx : (c == 1 ? ily : ilz)));
            const float e = d - box[3 + c][lane] - 1.0e-6f * (fabsf(m0) + fabsf(p) + box[3 + c][lane] + l);
            r2 += e > 0.f ? e * e : 0.f;
         }
         near = !(r2 > 1.00001f * cut2);
      }
      unsigned todo = __ballot_sync(0xffffffffu, near);
      while (todo) {
         float3 d[NA_STEP];
         unsigned in[NA_STEP];
         int at[NA_STEP];
#pragma unroll
         for (int u = 0; u < NA_STEP; ++u) {
            const bool some = todo != 0;
            at[u] = 32 * (some ? __ffs(todo) - 1 : 0) + lane;
            todo &= todo - 1;
            d[u].x = na_image(sx[3 * at[u]] - px, lx, ilx);
            d[u].y = na_image(sx[3 * at[u] + 1] - py, ly, ily);
            d[u].z = na_image(sx[3 * at[u] + 2] - pz, lz, ilz);
            const float r2 = d[u].x * d[u].x + d[u].y * d[u].y + d[u].z * d[u].z;
            in[u] = __ballot_sync(0xffffffffu, some && at[u] < m && !(r2 > cut2));
         }
#pragma unroll
         for (int u = 0; u < NA_STEP; ++u) {
            if (in[u] == 0)
               continue;
            if (in[u] >> lane & 1)
               ring[w][(tail + __popc(in[u] & lt)) & (NA_QUEUE - 1)] =
                  make_float4(d[u].x, d[u].y, d[u].z, __int_as_float(c0 + at[u]));
            tail += __popc(in[u]);
            if (tail - head >= 32) {
               __syncwarp();
               const float4 p = ring[w][(head + lane) & (NA_QUEUE - 1)];
               __syncwarp();
               head += 32;
               na_pair(p, i, pdi, pti, pdamp, thole, uind, uinp, f);
            }
         }
      }
   }
   __syncwarp();
   if (lane < tail - head)
      na_pair(ring[w][(head + lane) & (NA_QUEUE - 1)], i, pdi, pti, pdamp, thole, uind, uinp, f);
   __syncwarp();
   const float s = warp_sums<6>(f, lane);
   const int k = sum_slot<6>(lane);
   if (i < n && k >= 0)
      (k < 3 ? field : fieldp)[3 * i + k % 3] = s;
}

// do the two byte ranges share memory
static bool na_overlap(const void* a, size_t na, const void* b, size_t nb)
{
   const char *p = static_cast<const char*>(a), *q = static_cast<const char*>(b);
   return p < q + nb && q < p + na;
}

}  // namespace t9gb

extern "C" int t9gb_ufield_noalloc(int n, const double* box, double cutoff, const float* xyz, const float* pdamp,
   const float* thole, const float* uind, const float* uinp, float* field, float* fieldp, void* stream)
{
   using namespace t9gb;
   if (n <= 0 || !xyz || !pdamp || !thole || !uind || !uinp || !field || !fieldp || !(cutoff > 0))
      return T9GB_BAD_ARG;
   if (n > T9GB_NOALLOC_MAX_ATOMS)
      return T9GB_TOO_LARGE;
   int dev = 0;
   if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
      return T9GB_NO_DEVICE;
   const bool pbc = box && box[0] > 0 && box[1] > 0 && box[2] > 0;
   const float lx = pbc ? (float)box[0] : 0.f, ly = pbc ? (float)box[1] : 0.f, lz = pbc ? (float)box[2] : 0.f;
   const float ilx = pbc ? (float)(1.0 / box[0]) : 0.f, ily = pbc ? (float)(1.0 / box[1]) : 0.f;
   const float ilz = pbc ? (float)(1.0 / box[2]) : 0.f;
   const double c2 = cutoff * cutoff;
   const float cut2 = c2 > 3.0e38 ? 3.0e38f : (float)c2;
   cudaStream_t s = static_cast<cudaStream_t>(stream);
   // one launch unless an output overlaps an input
   const size_t b1 = sizeof(float) * n, b3 = 3 * b1;
   bool over = false;
   for (const float* o : {field, fieldp})
      over = over || na_overlap(o, b3, xyz, b3) || na_overlap(o, b3, uind, b3) || na_overlap(o, b3, uinp, b3) ||
         na_overlap(o, b3, pdamp, b1) || na_overlap(o, b3, thole, b1);
   if (over) {
      float* to = nullptr;
      const int rc = noalloc_scratch(dev, &to);
      if (rc != T9GB_OK)
         return rc;
      k_noalloc_copy<<<grid_for(3ll * n, 256), 256, 0, s>>>(n, xyz, pdamp, thole, uind, uinp, to);
      xyz = to, uind = to + 3 * n, uinp = to + 6 * n, pdamp = to + 9 * n, thole = to + 10 * n;
   }
   k_noalloc_ufield<<<grid_for(n, NA_WARPS), 32 * NA_WARPS, 0, s>>>(n, lx, ly, lz, ilx, ily, ilz, cut2,
      xyz, pdamp, thole, uind, uinp, field, fieldp);
   return cudaGetLastError() == cudaSuccess ? T9GB_OK : T9GB_CUDA_ERR;
}
