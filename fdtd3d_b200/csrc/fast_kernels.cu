// fast_kernels.cu - FP32 / FP16-storage form of the fdtd3d step, plus the
// conversion and reduction kernels.
//
// Formulation (algebraically the reference's, re-scaled and with the PML
// auxiliary fields kept only where sigma != 0):
//   H is stored as H' = eta0 * H, so with S = c*dt/dx every update reads
//     interior cells:  F += S / m * curl
//     PML cells:       X_new = ca1 * X + S * q1 * curl
//                      F     = p5 * F + (g4p * X_new - g4m * X) * q5 / m
//   where m is the averaged eps (E) or mu (H), X = D/eps0 or c*B, and the
//   1-D tables come from the reference's sigma profiles
//   (Source/Scheme/InternalScheme.inc.h:2297-2349, 2551-2640; the PML
//   coefficients of H use eps0 as in the reference).  In interior cells the
//   reference's D/B chain with sigma = 0 reduces exactly to the first line.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "cell_walk.cuh"
#include "kernels.h"

namespace fdtdb {

namespace {

template <typename T>
__device__ __forceinline__ float ld (const T *p, size_t i);
template <>
__device__ __forceinline__ float ld<float> (const float *p, size_t i)
{
  return p[i];
}
template <>
__device__ __forceinline__ float ld<__half> (const __half *p, size_t i)
{
  return __half2float (p[i]);
}

template <typename T>
__device__ __forceinline__ void st (T *p, size_t i, float v);
template <>
__device__ __forceinline__ void st<float> (float *p, size_t i, float v)
{
  p[i] = v;
}
template <>
__device__ __forceinline__ void st<__half> (__half *p, size_t i, float v)
{
  p[i] = __float2half_rn (v);
}

__device__ __forceinline__ size_t flin (const GeomDev &g, int x, int y, int z)
{
  return ((size_t) x * g.n[1] + y) * g.pz + z;
}

// incident value in FP64 (1-D grid is FP64 in every form)
__device__ __forceinline__ double fast_incident (const GeomDev &g, const double *inc, int inc_len, int *err, int k,
                                                 int px, int py, int pz)
{
  double d_diff = k >= 3 ? 0.5 : 0.0;
  double d;
  const int pos[3] = {px, py, pz};
  if (g.drop == 0)
  {
    double x = ((double) px + g.min_fp[k][0]) - g.zero_inc[0];
    double y = ((double) py + g.min_fp[k][1]) - g.zero_inc[1];
    double z = ((double) pz + g.min_fp[k][2]) - g.zero_inc[2];
    d = x * g.s1 * g.c2 + y * g.s1 * g.s2 + z * g.c1 - d_diff;
  }
  else
  {
    const int a0 = g.inc_ax[0], a1 = g.inc_ax[1];
    double u = ((double) pos[a0] + g.min_fp[k][a0]) - g.zero_inc[a0];
    double v = ((double) pos[a1] + g.min_fp[k][a1]) - g.zero_inc[a1];
    d = u * g.inc_k[0] + v * g.inc_k[1] - d_diff;
  }
  int i1 = (int) d;
  double pr2 = d - (double) i1;
  if (i1 < 0 || i1 + 1 >= inc_len)
  {
    if (err)
      *err = 1;
    return 0.0;
  }
  return (inc[i1] * (1 - pr2) + inc[i1 + 1] * pr2) * g.proj[k];
}

template <typename T>
__device__ __forceinline__ void fast_component (const FastHalf &p, int ci, int *err, int x, int y, int z)
{
  const GeomDev &g = p.g;
  const CompDev &c = p.comp[ci];
  const size_t id = flin (g, x, y, z);
  T *F = (T *) p.f[ci];
  const T *o1 = (const T *) p.opp[c.opp1];
  const T *o2 = (const T *) p.opp[c.opp2];
  float v0 = 0.f, v1 = 0.f, v2 = 0.f, v3 = 0.f;
  if (o1)
  {
    v0 = ld (o1, flin (g, x + c.d11[0], y + c.d11[1], z + c.d11[2]));
    v1 = ld (o1, flin (g, x + c.d12[0], y + c.d12[1], z + c.d12[2]));
  }
  if (o2)
  {
    v2 = ld (o2, flin (g, x + c.d21[0], y + c.d21[1], z + c.d21[2]));
    v3 = ld (o2, flin (g, x + c.d22[0], y + c.d22[1], z + c.d22[2]));
  }
  if (p.use_tfsf)
  {
    for (int t = 0; t < c.nterms; ++t)
    {
      const TermDev &tm = c.term[t];
      if (x >= tm.lo[0] && x < tm.hi[0] && y >= tm.lo[1] && y < tm.hi[1] && z >= tm.lo[2] && z < tm.hi[2])
      {
        double diff = fast_incident (g, p.inc, p.inc_len, err, tm.inc_comp, x + tm.aux[0], y + tm.aux[1],
                                     z + tm.aux[2]);
        float dv = (float) (diff * tm.negate) * p.inc_scale[tm.inc_comp];
        if (tm.slot == 0)
          v0 -= dv;
        else if (tm.slot == 1)
          v1 -= dv;
        else if (tm.slot == 2)
          v2 -= dv;
        else
          v3 -= dv;
      }
    }
  }
  float curl = (v1 - v0) - (v3 - v2);
  // J / M current source: the reference subtracts I dx Cb from the new D
  // (or E), i.e. I dx from the curl, here in the curl's scaled units
  if (((p.cs_mask >> ci) & 1) && x == p.cs[0] && y == p.cs[1] && z == p.cs[2])
    curl -= (float) (*p.cs_val * p.g.dx) * p.cs_scale;

  float inv_m = 1.f, m = 1.f;
  const float *mp = p.matc[ci] ? p.matc[ci] : p.mat;
  if (mp)
  {
    if (c.nmat == 1)
      m = mp[id];
    else if (c.nmat == 2)
      m = 0.5f * (mp[flin (g, x, y, z)] + mp[flin (g, x + c.m[1][0], y + c.m[1][1], z + c.m[1][2])]);
    else
      m = 0.25f * (mp[flin (g, x, y, z)] + mp[flin (g, x + c.m[1][0], y + c.m[1][1], z + c.m[1][2])]
                   + mp[flin (g, x + c.m[2][0], y + c.m[2][1], z + c.m[2][2])]
                   + mp[flin (g, x + c.m[3][0], y + c.m[3][1], z + c.m[3][2])]);
    inv_m = 1.f / m;
  }

  const int pos[3] = {x, y, z};
  bool interior = true;
  if (p.use_pml)
  {
#pragma unroll
    for (int a = 0; a < 3; ++a)
      interior = interior && pos[a] >= p.ilo[ci][a] && pos[a] < p.ihi[ci][a];
  }
  float f = ld (F, id);
  // Drude cell: a nonzero plasma frequency or collision rate on the
  // component's averaging stencil (getMetaMaterial: the mean of its two or
  // four points; metamaterials run with PML, as the reference's do)
  float w = 0.f, gm = 0.f;
  if (p.meta)
  {
    for (int j = 0; j < c.nmat; ++j)
    {
      const size_t q = flin (g, x + c.m[j][0], y + c.m[j][1], z + c.m[j][2]);
      w += p.om[q];
      gm += p.ga[q];
    }
    const float inv_n = c.nmat == 4 ? 0.25f : (c.nmat == 2 ? 0.5f : 1.f);
    w *= inv_n;
    gm *= inv_n;
  }
  if (p.meta && (w != 0.f || gm != 0.f))
  {
    // X by the curl step (PML coefficients; sigma = 0 gives ca1 = 1,
    // sq1 = S), the Drude recurrence to Z (the reference's b0 .. a2,
    // InternalScheme.inc.h:2527-2532, in the scaled units), F from Z with
    // material modifier 1 (InternalScheme.inc.h:2452-2640).  The recurrence
    // Z_n = b0 X_n + b1 X_o + b2 X_pp - a1 Z_o - a2 Z_pp is evaluated on
    // increments (b0 + b1 + b2 = 0 and 1 + a1 + a2 = 4 sq / A):
    //   dZ = b0 dX - b2 dX_o + a2 dZ_o - (4 sq / A) Z_o,
    // so that FP32 does not subtract nearly equal products of the fields;
    // this path keeps the last increments dX_o, dZ_o per cell (xpp, zpp).
    const int a0 = c.sig4, a1 = c.sig_cacb, a2 = c.sig5;
    const float ca1 = p.tab[ci][0][pos[a1]];
    const float sq1 = p.tab[ci][1][pos[a1]];
    const float p5 = p.tab[ci][2][pos[a2]];
    const float q5 = p.tab[ci][3][pos[a2]];
    const float g4p = p.tab[ci][4][pos[a0]];
    const float g4m = p.tab[ci][5][pos[a0]];
    float *X = p.aux[ci];
    const float xo = X[id], dxo = p.xpp[ci][id], zo = p.zd[ci][id], dzo = p.zpp[ci][id];
    const float dt = p.dt;
    const float sq = (dt * w) * (dt * w);
    const float inv = 1.f / (4.f * m + 2.f * dt * m * gm + sq);
    const float b0 = (4.f + 2.f * dt * gm) * inv, b2 = (4.f - 2.f * dt * gm) * inv;
    const float a2c = (4.f * m - 2.f * dt * m * gm + sq) * inv;
    const float dx = (ca1 - 1.f) * xo + sq1 * curl;
    const float dz = b0 * dx - b2 * dxo + a2c * dzo - (4.f * sq * inv) * zo;
    X[id] = xo + dx;
    p.xpp[ci][id] = dx;
    p.zd[ci][id] = zo + dz;
    p.zpp[ci][id] = dz;
    f = p5 * f + ((g4p - g4m) * zo + g4p * dz) * q5;
  }
  else if (interior)
  {
    f += p.courant * inv_m * curl;
  }
  else
  {
    const int a0 = c.sig4, a1 = c.sig_cacb, a2 = c.sig5;
    const float ca1 = p.tab[ci][0][pos[a1]];
    const float sq1 = p.tab[ci][1][pos[a1]];
    const float p5 = p.tab[ci][2][pos[a2]];
    const float q5 = p.tab[ci][3][pos[a2]];
    const float g4p = p.tab[ci][4][pos[a0]];
    const float g4m = p.tab[ci][5][pos[a0]];
    float *X = p.aux[ci];
    const float xo = X[id];
    const float xn = ca1 * xo + sq1 * curl;
    X[id] = xn;
    f = p5 * f + (g4p * xn - g4m * xo) * q5 * inv_m;
  }
  st (F, id, f);
}

// BLOCKS: CTAs an SM is to hold.  The kernel waits for memory, so large grids
// take six (40 registers, 44 B of spills) and grids that four hold at once
// four (59 registers, none).  us per step, left to the compiler (56 registers
// in FP16 storage, 48 in FP32) / now: H_CENTERED 200^3 FP16 617 / 506, FP32 504 /
// 489, 61^3 31.4 / 28.1, 30.3 / 27.4; 2-D with a DFT 2048^2 FP16 176 / 158.
template <typename T, int BLOCKS>
__global__ void __launch_bounds__ (256, BLOCKS) fast_half_kernel (FastHalf p, int *err)
{
  // interior cells: 1 .. n - 2 on every axis a mode keeps, 0 on a dropped one
  const int ix = (p.g.drop & 1) ? 1 : p.g.n[0] - 2;
  const int iy = (p.g.drop & 2) ? 1 : p.g.n[1] - 2;
  const int iz = (p.g.drop & 4) ? 1 : p.g.n[2] - 2;
  const int oz = (p.g.drop & 4) ? 0 : 1, oy = (p.g.drop & 2) ? 0 : 1, ox = (p.g.drop & 1) ? 0 : 1;
  for (CellWalk w ((int64_t) blockIdx.x * blockDim.x + threadIdx.x, (int64_t) gridDim.x * blockDim.x, ix, iy, iz);
       w.ok (); w.next ())
  {
    const int z = w.cz + oz, y = w.cy + oy, x = w.cx + ox;
#pragma unroll 1
    for (int ci = 0; ci < 3; ++ci)
    {
      if (p.comp[ci].exists)
        fast_component<T> (p, ci, err, x, y, z);
    }
  }
}

template <typename T>
__global__ void fast_point_source_kernel (T *f, size_t index, const double *src, int src_index, float scale)
{
  if (threadIdx.x == 0 && blockIdx.x == 0)
    st (f, index, (float) src[src_index] * scale);
}

// FP64 arrays <-> stored fields, dst = src * scale.  A copy is bound by DRAM
// (8 + sizeof (T) bytes per cell), so the flat form (rows without padding,
// both pointers on 16-byte boundaries) moves four cells per thread in 16-byte
// accesses where the grid is large (256^3 FP32 69 -> 58 us a call; with a
// quarter of the threads 4 M cells would take 31 instead of 28); the row form
// takes rows of nz cells, pz stored, a thread a cell.
__device__ __forceinline__ void ld4 (const double *p, size_t q, double v[4])
{
  const double2 a = reinterpret_cast<const double2 *> (p)[2 * q], b = reinterpret_cast<const double2 *> (p)[2 * q + 1];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}
__device__ __forceinline__ void ld4 (const float *p, size_t q, double v[4])
{
  const float4 a = reinterpret_cast<const float4 *> (p)[q];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
}
__device__ __forceinline__ void ld4 (const __half *p, size_t q, double v[4])
{
  const uint2 t = reinterpret_cast<const uint2 *> (p)[q];
  const float2 a = __half22float2 (*reinterpret_cast<const __half2 *> (&t.x));
  const float2 b = __half22float2 (*reinterpret_cast<const __half2 *> (&t.y));
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}
__device__ __forceinline__ void st4 (double *p, size_t q, const double v[4])
{
  __stcs (reinterpret_cast<double2 *> (p) + 2 * q, make_double2 (v[0], v[1]));
  __stcs (reinterpret_cast<double2 *> (p) + 2 * q + 1, make_double2 (v[2], v[3]));
}
__device__ __forceinline__ void st4 (float *p, size_t q, const double v[4])
{
  reinterpret_cast<float4 *> (p)[q] = make_float4 ((float) v[0], (float) v[1], (float) v[2], (float) v[3]);
}
__device__ __forceinline__ void st4 (__half *p, size_t q, const double v[4])
{
  __half2 a = __floats2half2_rn ((float) v[0], (float) v[1]), b = __floats2half2_rn ((float) v[2], (float) v[3]);
  uint2 t;
  t.x = *reinterpret_cast<unsigned *> (&a);
  t.y = *reinterpret_cast<unsigned *> (&b);
  reinterpret_cast<uint2 *> (p)[q] = t;
}

__device__ __forceinline__ double get (const double *p, size_t i)
{
  return p[i];
}
__device__ __forceinline__ double get (const float *p, size_t i)
{
  return (double) p[i];
}
__device__ __forceinline__ double get (const __half *p, size_t i)
{
  return (double) __half2float (p[i]);
}
__device__ __forceinline__ void put (double *p, size_t i, double v)
{
  p[i] = v;
}
__device__ __forceinline__ void put (float *p, size_t i, double v)
{
  p[i] = (float) v;
}
__device__ __forceinline__ void put (__half *p, size_t i, double v)
{
  p[i] = __float2half_rn ((float) v);
}

template <typename D, typename S, bool VEC>
__global__ void __launch_bounds__ (256) convert_flat_kernel (D *dst, const S *src, size_t n, double scale)
{
  const size_t t = (size_t) blockIdx.x * blockDim.x + threadIdx.x, step = (size_t) gridDim.x * blockDim.x;
  const size_t n4 = VEC ? n / 4 : 0;
  for (size_t q = t; q < n4; q += step)
  {
    double v[4];
    ld4 (src, q, v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] *= scale;
    st4 (dst, q, v);
  }
  for (size_t i = 4 * n4 + t; i < n; i += step)
    put (dst, i, get (src, i) * scale);
}

template <typename D, typename S>
__global__ void __launch_bounds__ (256) convert_rows_kernel (D *dst, const S *src, size_t rows, unsigned nz,
                                                             unsigned dpitch, unsigned spitch, double scale)
{
  // (a thread's place and its stride in rows and cells, divided once)
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const unsigned sr = step / nz, sz = step - sr * nz;
  unsigned z = t % nz;
  for (size_t r = t / nz; r < rows; r += sr)
  {
    put (dst, r * dpitch + z, get (src, r * spitch + z) * scale);
    z += sz;
    if (z >= nz)
    {
      z -= nz;
      ++r;
    }
  }
}

// Compensated FP64 accumulation: (s, c) += v with the rounding error of the
// sum kept in c (Knuth's two-sum: no branch on the magnitudes).
__device__ __forceinline__ void two_sum (double &s, double &c, double v)
{
  const double t = s + v, z = t - s;
  c += (s - (t - z)) + (v - z);
  s = t;
}

// The (s, c) pairs of a warp's lanes added up in lane 0.
__device__ __forceinline__ void warp_sum (double &s, double &c)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    const double os = __shfl_down_sync (0xffffffffu, s, o), oc = __shfl_down_sync (0xffffffffu, c, o);
    two_sum (s, c, os);
    c += oc;
  }
}

// Block `part` of `parts` (256 threads each) of sum w v^2 scale over n values
// into partials[2 part], [2 part + 1].  Bound by the FP64 pipe (about ten
// instructions per value): two accumulators per thread hide their latency,
// and the block's pairs meet in a shuffle tree (a loop over 256 pairs in one
// thread, and one over the blocks in reduce_final, took more time than the
// sum: 55 MB 57 + 63 us before).
template <typename T>
__device__ __forceinline__ void reduce_block (const T *src, size_t n, const void *weight, int wkind, double scale,
                                              int part, int parts, double *partials)
{
  double s0 = 0.0, c0 = 0.0, s1 = 0.0, c1 = 0.0;
  auto term = [&] (size_t i) {
    const double v = get (src, i);
    const double w = wkind == 1 ? (double) ((const float *) weight)[i] : (wkind == 2 ? ((const double *) weight)[i] : 1.0);
    return w * v * v * scale;
  };
  const size_t step = (size_t) parts * 256;
  size_t i = (size_t) part * 256 + threadIdx.x;
  for (; i + step < n; i += 2 * step)
  {
    const double a = term (i), b = term (i + step);
    two_sum (s0, c0, a);
    two_sum (s1, c1, b);
  }
  if (i < n)
    two_sum (s0, c0, term (i));
  two_sum (s0, c0, s1);
  c0 += c1;
  warp_sum (s0, c0);
  __shared__ double sh[2][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0)
  {
    sh[0][w] = s0;
    sh[1][w] = c0;
  }
  __syncthreads ();
  if (w == 0)
  {
    s0 = lane < 8 ? sh[0][lane] : 0.0;
    c0 = lane < 8 ? sh[1][lane] : 0.0;
    warp_sum (s0, c0);
    if (lane == 0)
    {
      partials[2 * part] = s0;
      partials[2 * part + 1] = c0;
    }
  }
}

// One warp: the blocks' pairs into one value.
__device__ __forceinline__ void reduce_parts (const double *partials, int parts, double *out)
{
  double s = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < parts; i += 32)
  {
    two_sum (s, c, partials[2 * i]);
    c += partials[2 * i + 1];
  }
  warp_sum (s, c);
  if (threadIdx.x == 0)
    *out = s + c;
}

template <int KIND>
__global__ void __launch_bounds__ (256) reduce_sq_kernel (const void *src, size_t n, const void *weight,
                                                          int wkind, double scale, double *partials)
{
  using T = typename std::conditional<KIND == 0, double, typename std::conditional<KIND == 1, float, __half>::type>::type;
  reduce_block ((const T *) src, n, weight, wkind, scale, blockIdx.x, gridDim.x, partials);
}

__global__ void reduce_final_kernel (const double *partials, int nblocks, double *out)
{
  reduce_parts (partials, nblocks, out);
}

// every component in one launch: block row y takes item y
template <int KIND>
__global__ void __launch_bounds__ (256) reduce_items_kernel (const __grid_constant__ ReduceItems it, size_t n,
                                                             double *partials)
{
  using T = typename std::conditional<KIND == 0, double, typename std::conditional<KIND == 1, float, __half>::type>::type;
  const int q = blockIdx.y;
  reduce_block ((const T *) it.src[q], n, it.weight[q], it.wkind[q], it.scale[q], blockIdx.x, gridDim.x,
                partials + (size_t) 2 * gridDim.x * q);
}

__global__ void reduce_items_final_kernel (const __grid_constant__ ReduceItems it, const double *partials, int nblocks,
                                           double *out)
{
  reduce_parts (partials + (size_t) 2 * nblocks * blockIdx.x, nblocks, out + it.out[blockIdx.x]);
}

int grid_for (size_t n, int sm_count)
{
  size_t b = (n + 255) / 256;
  size_t cap = (size_t) sm_count * 16;
  if (b > cap)
    b = cap;
  return b < 1 ? 1 : (int) b;
}

}  // namespace

int launch_fast_half (const FastHalf &p, int *err, int sm_count, cudaStream_t s)
{
  const int ix = (p.g.drop & 1) ? 1 : p.g.n[0] - 2;
  const int iy = (p.g.drop & 2) ? 1 : p.g.n[1] - 2;
  const int iz = (p.g.drop & 4) ? 1 : p.g.n[2] - 2;
  int64_t total = (int64_t) ix * iy * iz;
  int64_t blocks = (total + 255) / 256;
  int64_t cap = (int64_t) sm_count * 8 * 16;
  if (blocks > cap)
    blocks = cap;
  if (blocks < 1)
    blocks = 1;
  const bool few = blocks <= 4 * (int64_t) sm_count;
  auto kern = p.fp16 ? (few ? fast_half_kernel<__half, 4> : fast_half_kernel<__half, 6>)
                     : (few ? fast_half_kernel<float, 4> : fast_half_kernel<float, 6>);
  kern<<<(unsigned) blocks, 256, 0, s>>> (p, err);
  return 1;
}

int launch_fast_point_source (void *f, int fp16, size_t index, const double *src, int src_index, float scale,
                              cudaStream_t s)
{
  if (fp16)
    fast_point_source_kernel<__half><<<1, 32, 0, s>>> ((__half *) f, index, src, src_index, scale);
  else
    fast_point_source_kernel<float><<<1, 32, 0, s>>> ((float *) f, index, src, src_index, scale);
  return 1;
}

namespace {

template <typename D, typename S>
int launch_convert (D *dst, const S *src, size_t rows, int nz, int dpitch, int spitch, double scale, cudaStream_t s)
{
  if (nz == dpitch && nz == spitch)
  {
    const size_t n = rows * (size_t) nz;
    const bool vec = n >= (size_t) 8000000 && (((uintptr_t) dst | (uintptr_t) src) & 15u) == 0;
    if (vec)
      convert_flat_kernel<D, S, true><<<grid_for ((n + 3) / 4, 148), 256, 0, s>>> (dst, src, n, scale);
    else
      convert_flat_kernel<D, S, false><<<grid_for (n, 148), 256, 0, s>>> (dst, src, n, scale);
  }
  else
    convert_rows_kernel<<<grid_for (rows * (size_t) nz, 148), 256, 0, s>>> (dst, src, rows, nz, dpitch, spitch, scale);
  return 1;
}

}  // namespace

int launch_convert_in (void *dst, int dst_kind, const double *src, size_t rows, int nz, int pz, double scale,
                       cudaStream_t s)
{
  if (dst_kind == 0)
    return launch_convert ((double *) dst, src, rows, nz, pz, nz, scale, s);
  if (dst_kind == 1)
    return launch_convert ((float *) dst, src, rows, nz, pz, nz, scale, s);
  return launch_convert ((__half *) dst, src, rows, nz, pz, nz, scale, s);
}

namespace {

// lowest index of a non-finite value (NaN or +-Inf) into *first
__global__ void find_nonfinite_kernel (const double *src, size_t n, unsigned long long *first)
{
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x)
    if (!isfinite (src[i]))
      atomicMin (first, (unsigned long long) i);
}

}  // namespace

int launch_find_nonfinite (const double *src, size_t n, unsigned long long *first, cudaStream_t s)
{
  find_nonfinite_kernel<<<grid_for (n, 148), 256, 0, s>>> (src, n, first);
  return 1;
}

int launch_convert_out (double *dst, const void *src, int src_kind, size_t rows, int nz, int pz, double scale,
                        cudaStream_t s)
{
  if (src_kind == 0)
    return launch_convert (dst, (const double *) src, rows, nz, nz, pz, scale, s);
  if (src_kind == 1)
    return launch_convert (dst, (const float *) src, rows, nz, nz, pz, scale, s);
  return launch_convert (dst, (const __half *) src, rows, nz, nz, pz, scale, s);
}

int launch_reduce_items (const ReduceItems &it, int kind, size_t n, double *partials, int nblocks, double *out,
                         cudaStream_t s)
{
  if (it.count == 0)
    return 0;
  const dim3 grid (nblocks, it.count);
  if (kind == 0)
    reduce_items_kernel<0><<<grid, 256, 0, s>>> (it, n, partials);
  else if (kind == 1)
    reduce_items_kernel<1><<<grid, 256, 0, s>>> (it, n, partials);
  else
    reduce_items_kernel<2><<<grid, 256, 0, s>>> (it, n, partials);
  reduce_items_final_kernel<<<it.count, 32, 0, s>>> (it, partials, nblocks, out);
  return 2;
}

__global__ void fill_kernel (double *dst, size_t n, double value)
{
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x)
    dst[i] = value;
}

int launch_fill (double *dst, size_t n, double value, cudaStream_t s)
{
  fill_kernel<<<grid_for (n, 148), 256, 0, s>>> (dst, n, value);
  return 1;
}

// The allocation-free sum's two launches through cudaLaunchKernel, so that
// each returns its own launch status and an earlier, unrelated error pending on the calling
// thread is neither reported nor cleared.
cudaError_t launch_reduce_sq_checked (const void *src, int kind, size_t n, const void *weight, int wkind,
                                      double scale, double *partials, int nblocks, cudaStream_t s)
{
  const void *fn = kind == 0 ? (const void *) reduce_sq_kernel<0>
                   : kind == 1 ? (const void *) reduce_sq_kernel<1>
                               : (const void *) reduce_sq_kernel<2>;
  void *args[] = {(void *) &src, (void *) &n, (void *) &weight, (void *) &wkind, (void *) &scale,
                  (void *) &partials};
  return cudaLaunchKernel (fn, dim3 (nblocks), dim3 (256), args, 0, s);
}

cudaError_t launch_reduce_final_checked (const double *partials, int nblocks, double *out, cudaStream_t s)
{
  void *args[] = {(void *) &partials, (void *) &nblocks, (void *) &out};
  return cudaLaunchKernel ((const void *) reduce_final_kernel, dim3 (1), dim3 (32), args, 0, s);
}

}  // namespace fdtdb

// ------------------------------------------------------------ running DFT

namespace fdtdb {

namespace {

__device__ __forceinline__ double ldd (const double *p, size_t i)
{
  return p[i];
}
__device__ __forceinline__ double ldd (const float *p, size_t i)
{
  return (double) p[i];
}
__device__ __forceinline__ double ldd (const __half *p, size_t i)
{
  return (double) __half2float (p[i]);
}

__device__ __forceinline__ void neumaier (double *s, double *c, double v)
{
  const double t = *s + v;
  if (fabs (*s) >= fabs (v))
    *c += (*s - t) + v;
  else
    *c += (v - t) + *s;
  *s = t;
}

// One time step of the running DFT of a stored field on the plane
// x_axis = index: for every plane cell and frequency j,
//   sum_j += v * exp(-i phase_j),  phase table = (cos, sin) per frequency,
// in FP64 with Neumaier compensation (acc: re, re compensation, im, im
// compensation per cell and frequency).
template <typename T>
__global__ void dft_kernel (const T *src, int axis, int index, int n0, int n1, int n2, int pz, double scale,
                            const double *phase, int nf, double *acc)
{
  const int ma = axis == 0 ? n1 : n0;             // plane extents (first, second remaining axis)
  const int mb = axis == 2 ? n1 : n2;
  const long long cells = (long long) ma * mb;
  for (long long q = (long long) blockIdx.x * blockDim.x + threadIdx.x; q < cells * nf;
       q += (long long) gridDim.x * blockDim.x)
  {
    const int j = (int) (q / cells);
    const long long c = q % cells;
    const int a = (int) (c / mb), b = (int) (c % mb);
    long long id;
    if (axis == 0)
      id = ((long long) index * n1 + a) * pz + b;
    else if (axis == 1)
      id = ((long long) a * n1 + index) * pz + b;
    else
      id = ((long long) a * n1 + b) * pz + index;
    const double v = ldd (src, (size_t) id) * scale;
    double *r = acc + q * 4;
    neumaier (r + 0, r + 1, v * phase[2 * j]);
    neumaier (r + 2, r + 3, -v * phase[2 * j + 1]);
  }
}

}  // namespace

int launch_dft (const void *src, int kind, int axis, int index, const int n[3], int pz, double scale,
                const double *phase, int nf, double *acc, int sm_count, cudaStream_t s)
{
  const long long cells = (long long) (axis == 0 ? n[1] : n[0]) * (axis == 2 ? n[1] : n[2]) * nf;
  long long blocks = (cells + 255) / 256;
  if (blocks > (long long) sm_count * 16)
    blocks = (long long) sm_count * 16;
  if (kind == 0)
    dft_kernel<double><<<(unsigned) blocks, 256, 0, s>>> ((const double *) src, axis, index, n[0], n[1], n[2], pz, scale,
                                                          phase, nf, acc);
  else if (kind == 1)
    dft_kernel<float><<<(unsigned) blocks, 256, 0, s>>> ((const float *) src, axis, index, n[0], n[1], n[2], pz, scale,
                                                         phase, nf, acc);
  else
    dft_kernel<__half><<<(unsigned) blocks, 256, 0, s>>> ((const __half *) src, axis, index, n[0], n[1], n[2], pz, scale,
                                                          phase, nf, acc);
  return 1;
}

}  // namespace fdtdb
