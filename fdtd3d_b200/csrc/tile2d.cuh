// tile2d.cuh - several time steps of a 2-D mode in one launch, for the FP64
// plain form (compiled with --fmad=false) and the FP32 / FP16-storage forms.
//
// A 2-D step is a chain of tiny dependent launches (E, H, two incident-grid
// steps, sources): 512^2 cells in FP32 took 24 us per step and 120 x 100 in
// FP64 21 us, all launch and L2 latency.  Here a CTA takes a tile with a halo
// of kTileSteps cells, keeps its cells' fields in registers and the current
// level in shared memory for the neighbours, and advances up to kTileSteps
// steps with one __syncthreads per half-step; the halo's values are computed
// twice instead of exchanged, one cell of it turning invalid per step.  Every
// cell's arithmetic is the per-cell kernels', so FP64 fields keep their bits;
// FP16 storage rounds once per launch instead of once per half-step.  A run
// of 100 steps at 120 x 100 in FP64, its three fields read by the host: 2133
// -> 655 us; 200 steps at 512^2 in FP32: 4820 -> 2330 us (of which the host
// copies are about 900).
// The part of the 1-D incident grid a tile's TF/SF terms can reach advances
// in shared memory with it; a few CTAs advance the whole grid.
// FP64 keeps two levels of every field whose face cells are never updated: a
// step leaves the other level's face cells current, so a tile alternates the
// two values, and an odd number of steps per launch ends on the level that
// is written.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>

#include "tile2d.h"

namespace fdtdb {

namespace {

constexpr int kTileWarps = 16;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kWindow = 192;        // incident cells a tile can reach: 66 sqrt 2 + 2 kTileSteps + margins
constexpr int kSrcRow = 5;          // doubles per step in the source table
constexpr int kIncOwn = kTileThreads - 2 * kTileSteps;

__device__ __forceinline__ double tile_ld (const double *p, int64_t i) { return p[i]; }
__device__ __forceinline__ float tile_ld (const float *p, int64_t i) { return p[i]; }
__device__ __forceinline__ float tile_ld (const __half *p, int64_t i) { return __half2float (p[i]); }
__device__ __forceinline__ void tile_st (double *p, int64_t i, double v) { p[i] = v; }
__device__ __forceinline__ void tile_st (float *p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void tile_st (__half *p, int64_t i, float v) { p[i] = __float2half_rn (v); }

// The incident grid on [c0, c0 + n) in shared memory: E, then H step.  Cells
// whose neighbour lies outside the window turn invalid from its ends inwards.
__device__ __forceinline__ void inc_e_step (double *e, const double *h, int c0, int n, const Tile2D &p, double src)
{
  const int q = threadIdx.x + 32 * threadIdx.y, i = c0 + q;
  if (q < n && i < p.inc_len)
  {
    if (i == 0)
      e[q] = src;
    else if (q > 0)
      e[q] = e[q] + (h[q - 1] - h[q]) * p.mod_e;
  }
}
__device__ __forceinline__ void inc_h_step (double *h, const double *e, int c0, int n, const Tile2D &p)
{
  const int q = threadIdx.x + 32 * threadIdx.y, i = c0 + q;
  if (q + 1 < n && i < p.inc_len - 1)
    h[q] = h[q] + (e[q] - e[q + 1]) * p.mod_h;
}

// Incident value of absolute component k at cell (u, v), from the window.
__device__ __forceinline__ double tile_incident (const Tile2D &p, const double *win, int c0, int k, int u, int v)
{
  const double du = ((double) u + p.pos[k][0]) - p.zero[0];
  const double dv = ((double) v + p.pos[k][1]) - p.zero[1];
  const double d = du * p.k[0] + dv * p.k[1] - (k >= 3 ? 0.5 : 0.0);
  const double cd1 = (double) ((int) d);
  const double pr2 = d - cd1, pr1 = 1 - pr2;
  const int i1 = (int) cd1, q = i1 - c0;
  if (i1 < 0 || i1 + 1 >= p.inc_len || q < 0 || q + 1 >= kWindow)
  {
    *p.err = 1;
    return 0.0;
  }
  return (win[q] * pr1 + win[q + 1] * pr2) * p.proj[k];
}

// Compile-time structure of a mode (FORM = te + 2 flip + 4 hc).  Axes: 0 u,
// 1 v, 2 the dropped one (w).  Component a of E has the curl differences
// H_{a+2} along a + 1 and H_{a+1} along a + 2, of H E_{a+1} along a + 2 and
// E_{a+2} along a + 1 (a + 1, a + 2: cyclic); PML pairs: curl step along
// a + 1, field along a + 2, auxiliary along a.
template <int FORM>
struct Mode2D
{
  static constexpr bool TE = FORM & 1, FLIP = FORM & 2, HC = FORM & 4;
  static constexpr int axis (int j) { return TE ? (j < 2 ? j : 2) : (j == 0 ? 2 : j - 1); }
  static constexpr bool is_h (int j) { return TE ? j == 2 : j > 0; }
  static constexpr int next (int a) { return (a + (FLIP ? 2 : 1)) % 3; }
  // slot of the component of a family along axis a, -1: not in the mode
  static constexpr int slot (bool h, int a) { return TE ? (h ? (a == 2 ? 2 : -1) : (a < 2 ? a : -1)) : (h ? (a < 2 ? 1 + a : -1) : (a == 2 ? 0 : -1)); }
  static constexpr int opp (int j, int q)
  {
    const int n = next (axis (j)), m = next (n);
    return slot (!is_h (j), is_h (j) == (q == 0) ? n : m);
  }
  static constexpr int along (int j, int q)
  {
    const int n = next (axis (j)), m = next (n);
    return is_h (j) == (q == 0) ? m : n;
  }
  static constexpr int low (int j) { return is_h (j) == HC ? -1 : 0; }
  static constexpr int ax1 (int j) { return next (axis (j)); }
  static constexpr int ax5 (int j) { return next (next (axis (j))); }
  static constexpr int ax4 (int j) { return axis (j); }
};

// Shared memory of a tile, in values of the arithmetic type: the fields with a
// border of one cell, per-cell coefficients (FP64: E-from-D's two, or without
// PML the curl's; FP32: S / m) and the 1-D PML tables along the tile.
template <typename C, int CU, int CV>
struct TileMem
{
  static constexpr int TU = kTileWarps * CU, TV = 32 * CV, TM = TU > TV ? TU : TV;
  static constexpr int P = TV + 2, A = (TU + 2) * P, N = TU * TV;
  static constexpr int COEF = 3 * A, TAB = COEF + (sizeof (C) == 8 ? 6 : 3) * N;
  static constexpr int BYTES = (TAB + 3 * 6 * TM) * (int) sizeof (C);
};

// T: stored field type, C: arithmetic (double or float).  A thread holds the
// CU x CV cells (w + 16 j, lane + 32 i) of the 16 CU x 32 CV tile.
template <typename T, typename C, int CU, int CV, int FORM>
__global__ void __launch_bounds__ (kTileThreads, CU * CV > 2 ? 1 : 2) tile2d_kernel (const __grid_constant__ Tile2D p, int tiles_v,
                                                               int ntiles)
{
  constexpr bool F64 = sizeof (C) == 8;
  using L = TileMem<C, CU, CV>;
  using M = Mode2D<FORM>;
  constexpr int TU = L::TU, TV = L::TV, TM = L::TM, R = CU * CV, P = L::P, A = L::A, N = L::N;
  constexpr int OU = TU - 2 * kTileSteps, OV = TV - 2 * kTileSteps;
  extern __shared__ __align__ (16) unsigned char tile_smem[];
  C *const F = reinterpret_cast<C *> (tile_smem), *const K = F + L::COEF, *const Tab = F + L::TAB;
  __shared__ double s_inc[2][kTileThreads];
  const int lane = threadIdx.x, w = threadIdx.y;

  if ((int) blockIdx.x >= ntiles)
  {
    // a stretch of the incident grid
    const int c0 = ((int) blockIdx.x - ntiles) * kIncOwn - kTileSteps, q = lane + 32 * w, i = c0 + q;
    const bool in = i >= 0 && i < p.inc_len;
    s_inc[0][q] = in ? p.e_in[i] : 0.0;
    s_inc[1][q] = in ? p.h_in[i] : 0.0;
    __syncthreads ();
    for (int s = 0; s < p.steps; ++s)
    {
      if (i >= 0)
        inc_e_step (s_inc[0], s_inc[1], c0, kTileThreads, p, p.src[kSrcRow * s]);
      __syncthreads ();
      if (i >= 0)
        inc_h_step (s_inc[1], s_inc[0], c0, kTileThreads, p);
      __syncthreads ();
    }
    if (in && q >= kTileSteps && q < kTileThreads - kTileSteps && i < p.inc_cells)
    {
      p.e_out[i] = s_inc[0][q];
      p.h_out[i] = s_inc[1][q];
    }
    return;
  }

  const int u0 = ((int) blockIdx.x / tiles_v) * OU - kTileSteps, v0 = ((int) blockIdx.x % tiles_v) * OV - kTileSteps;
  for (int q = lane + 32 * w; q < 3 * A; q += kTileThreads)
    F[q] = C (0);

  if (p.use_pml)
    for (int q = lane + 32 * w; q < 3 * 6 * TM; q += kTileThreads)
    {
      const int j = q / (6 * TM), t = (q / TM) % 6, i = q % TM;
      const TileComp &c = p.comp[j];
      const int ax = t < 2 ? M::ax1 (j) : (t < 4 ? M::ax5 (j) : M::ax4 (j));
      const int g = ax == 0 ? u0 + i : (ax == 1 ? v0 + i : 0), n = ax == 0 ? p.nu : (ax == 1 ? p.nv : 1);
      Tab[q] = g >= 0 && g < n ? ((const C *) c.tab[t])[g] : C (1);
    }

  // ---- this thread's cells: field and PML auxiliary.  (FP64 face cells keep
  // the other level's field in the auxiliary's place, which they do not have.)
  C f[3][R], x[3][R];
  unsigned upd = 0, face = 0, source = 0, in_pml[3] = {0, 0, 0}, terms[R];
  bool any_term = false;
#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const int du = w + kTileWarps * (r / CV), dv = lane + 32 * (r % CV);
    const int u = u0 + du, v = v0 + dv;
    const bool valid = u >= 0 && u < p.nu && v >= 0 && v < p.nv;
    const bool up = u >= 1 && u <= p.nu - 2 && v >= 1 && v <= p.nv - 2;
    const int64_t id = (int64_t) u * p.nv + v;
    upd |= up ? 1u << r : 0u;
    face |= valid && !up ? 1u << r : 0u;
    source |= up && u == p.pu && v == p.pv ? 1u << r : 0u;
    terms[r] = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
      const TileComp &c = p.comp[j];
      f[j][r] = valid ? C (tile_ld ((const T *) c.in, id)) : C (0);
      x[j][r] = F64 && valid && !up ? C (tile_ld ((const T *) c.out, id)) : C (0);
      if (!up)
        continue;
      C m = C (1);
      if (c.mat)
      {
        C pt[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          pt[q] = q < c.nmat ? ((const C *) c.mat)[id + (int64_t) c.m[q][0] * p.nv + c.m[q][1]] : C (0);
        if constexpr (F64)
          m = c.nmat == 1 ? pt[0]
                          : (c.nmat == 2 ? (pt[0] + pt[1]) / 2.0
                                         : ((pt[0] + pt[1]) / 2.0 + (pt[2] + pt[3]) / 2.0) / 2.0);
        else
          m = c.nmat == 1 ? pt[0] : (c.nmat == 2 ? C (0.5) * (pt[0] + pt[1]) : C (0.25) * (pt[0] + pt[1] + pt[2] + pt[3]));
      }
      const int at = j * N + du * TV + dv;
      if constexpr (F64)
      {
        const double mm = p.mm[M::is_h (j)];
        if (p.use_pml)
        {
          x[j][r] = ((const C *) c.aux_in)[id];
          const C *const *tab = (const C *const *) c.tab;
          const int q5 = M::ax5 (j) == 0 ? u : (M::ax5 (j) == 1 ? v : 0);
          const int q4 = M::ax4 (j) == 0 ? u : (M::ax4 (j) == 1 ? v : 0);
          const double modifier = m * mm, dd = tab[3][q5], plus = tab[4][q4], minus = tab[5][q4];
          const double cp = (plus / modifier) / dd;
          K[at] = cp;
          K[3 * N + at] = minus == plus ? cp : (minus / modifier) / dd;
        }
        else
          K[at] = p.dt / (m * mm * p.dx);
      }
      else
      {
        K[at] = p.courant * (1.f / m);
        if (p.use_pml && !(u >= c.ilo[0] && u < c.ihi[0] && v >= c.ilo[1] && v < c.ihi[1]))
        {
          in_pml[j] |= 1u << r;
          x[j][r] = ((const float *) c.aux_in)[id];
          K[at] = 1.f / m;
        }
      }
      if (p.use_tfsf)
        for (int t = 0; t < c.nterms; ++t)
          if (u >= c.term[t].lo[0] && u < c.term[t].hi[0] && v >= c.term[t].lo[1] && v < c.term[t].hi[1])
            terms[r] |= 1u << (4 * j + t);
    }
    any_term |= terms[r] != 0;
  }
  // window of the incident grid the tile's terms reach during the steps
  int wc = 0;
  const bool tile_terms = __syncthreads_or (any_term ? 1 : 0) != 0;   // (also: the zeroed shared fields)
  if (tile_terms)
  {
    const double a0 = ((double) (u0 - 1) - p.zero[0]) * p.k[0], a1 = ((double) (u0 + TU + 1) - p.zero[0]) * p.k[0];
    const double b0 = ((double) (v0 - 1) - p.zero[1]) * p.k[1], b1 = ((double) (v0 + TV + 1) - p.zero[1]) * p.k[1];
    wc = max (0, (int) (fmin (a0, a1) + fmin (b0, b1)) - kTileSteps - 3);
    const int q = lane + 32 * w, i = wc + q;
    if (q < kWindow)
    {
      s_inc[0][q] = i < p.inc_len ? p.e_in[i] : 0.0;
      s_inc[1][q] = i < p.inc_len ? p.h_in[i] : 0.0;
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      F[j * A + (1 + w + kTileWarps * (r / CV)) * P + 1 + lane + 32 * (r % CV)] = f[j][r];
  __syncthreads ();

  for (int s = 0; s < p.steps; ++s)
  {
#pragma unroll
    for (int fam = 0; fam < 2; ++fam)
    {
      // the incident grid's half-step touches the family the terms do not
      // read: E terms read HInc before its update, H terms EInc after its
      if (tile_terms)
      {
        if (fam == 0)
          inc_e_step (s_inc[0], s_inc[1], wc, kWindow, p, p.src[kSrcRow * s]);
        else
          inc_h_step (s_inc[1], s_inc[0], wc, kWindow, p);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j)
      {
        const TileComp &c = p.comp[j];
        if (M::is_h (j) != (fam == 1))
          continue;
        constexpr int kStep[3] = {P, 1, 0};
        const int s1 = M::opp (j, 0), s2 = M::opp (j, 1);
        const int n11 = M::low (j) * kStep[M::along (j, 0)], n12 = n11 + kStep[M::along (j, 0)];
        const int n21 = M::low (j) * kStep[M::along (j, 1)], n22 = n21 + kStep[M::along (j, 1)];
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
          const int at = (1 + w + kTileWarps * (r / CV)) * P + 1 + lane + 32 * (r % CV);
          if ((upd >> r) & 1u)
          {
            C a = C (0), b = C (0), d = C (0), e = C (0);
            if (s1 >= 0)
            {
              a = F[s1 * A + at + n11];
              b = F[s1 * A + at + n12];
            }
            if (s2 >= 0)
            {
              d = F[s2 * A + at + n21];
              e = F[s2 * A + at + n22];
            }
            if (unsigned on = (terms[r] >> (4 * j)) & 15u)
            {
              const int u = u0 + w + kTileWarps * (r / CV), v = v0 + lane + 32 * (r % CV);
              for (; on; on &= on - 1)
              {
                const TermDev &tm = c.term[__ffs ((int) on) - 1];
                const double diff = tile_incident (p, s_inc[fam == 0 ? 1 : 0], wc, tm.inc_comp, u + tm.aux[0], v + tm.aux[1])
                                    * tm.negate;
                const C y = F64 ? C (diff) : C ((float) diff * p.scale[tm.inc_comp >= 3 ? 1 : 0]);
                a -= tm.slot == 0 ? y : C (0);
                b -= tm.slot == 1 ? y : C (0);
                d -= tm.slot == 2 ? y : C (0);
                e -= tm.slot == 3 ? y : C (0);
              }
            }
            const int du = w + kTileWarps * (r / CV), dv = lane + 32 * (r % CV);
            const C *const t = Tab + 6 * j * TM;
            const int q1 = M::ax1 (j) == 0 ? du : (M::ax1 (j) == 1 ? dv : 0);
            const int q5 = M::ax5 (j) == 0 ? du : (M::ax5 (j) == 1 ? dv : 0);
            const C kc = K[j * N + du * TV + dv];
            if constexpr (F64)
            {
              const C tmp = b - a - e + d;
              if (p.use_pml)
              {
                const C nx = x[j][r] * t[q1] + tmp * t[TM + q1];
                f[j][r] = f[j][r] * t[2 * TM + q5] + nx * kc - x[j][r] * K[(3 + j) * N + du * TV + dv];
                x[j][r] = nx;
              }
              else
                f[j][r] = f[j][r] + tmp * kc;
            }
            else
            {
              const C curl = (b - a) - (e - d);
              if ((in_pml[j] >> r) & 1u)
              {
                const int q4 = M::ax4 (j) == 0 ? du : (M::ax4 (j) == 1 ? dv : 0);
                const C nx = t[q1] * x[j][r] + t[TM + q1] * curl;
                f[j][r] = t[2 * TM + q5] * f[j][r]
                          + (t[4 * TM + q4] * nx - t[5 * TM + q4] * x[j][r]) * t[3 * TM + q5] * kc;
                x[j][r] = nx;
              }
              else
                f[j][r] += kc * curl;
            }
            if (((source >> r) & 1u) && c.source)
              f[j][r] = F64 ? C (p.src[kSrcRow * s + 1 + fam]) : C ((float) p.src[kSrcRow * s + 1 + fam] * p.scale[fam]);
          }
          else if (F64 && ((face >> r) & 1u))
          {
            const C t = f[j][r];
            f[j][r] = x[j][r];
            x[j][r] = t;
          }
          F[j * A + at] = f[j][r];
        }
      }
      __syncthreads ();
    }
  }

#pragma unroll
  for (int r = 0; r < R; ++r)
  {
    const int du = w + kTileWarps * (r / CV), dv = lane + 32 * (r % CV);
    if (!((upd >> r) & 1u) || du < kTileSteps || du >= TU - kTileSteps || dv < kTileSteps || dv >= TV - kTileSteps)
      continue;
    const int64_t id = (int64_t) (u0 + du) * p.nv + v0 + dv;
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
      tile_st ((T *) p.comp[j].out, id, f[j][r]);
      if (p.use_pml && (F64 || ((in_pml[j] >> r) & 1u)))
        ((C *) p.comp[j].aux_out)[id] = x[j][r];
    }
  }
}

template <typename T, typename C, int CU, int CV, int FORM>
int tile2d_start (const Tile2D &p, cudaStream_t s)
{
  constexpr int OU = kTileWarps * CU - 2 * kTileSteps, OV = 32 * CV - 2 * kTileSteps;
  constexpr int smem = TileMem<C, CU, CV>::BYTES;
  const int tu = (p.nu + OU - 1) / OU, tv = (p.nv + OV - 1) / OV;
  const int inc = p.use_tfsf ? (p.inc_cells + kIncOwn - 1) / kIncOwn : 0;
  auto kern = tile2d_kernel<T, C, CU, CV, FORM>;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  kern<<<tu * tv + inc, dim3 (32, kTileWarps), smem, s>>> (p, tv, tu * tv);
  return 1;
}

template <typename T, typename C, int CU, int CV>
int tile2d_launch (const Tile2D &p, cudaStream_t s)
{
  switch ((p.form.te ? 1 : 0) + (p.form.flip ? 2 : 0) + (p.form.hc ? 4 : 0))
  {
    case 0: return tile2d_start<T, C, CU, CV, 0> (p, s);
    case 1: return tile2d_start<T, C, CU, CV, 1> (p, s);
    case 2: return tile2d_start<T, C, CU, CV, 2> (p, s);
    case 3: return tile2d_start<T, C, CU, CV, 3> (p, s);
    case 4: return tile2d_start<T, C, CU, CV, 4> (p, s);
    case 5: return tile2d_start<T, C, CU, CV, 5> (p, s);
    case 6: return tile2d_start<T, C, CU, CV, 6> (p, s);
    default: return tile2d_start<T, C, CU, CV, 7> (p, s);
  }
}

// Tiles of a launch for a tile of CU x CV cells per thread.
inline int64_t tile2d_count (const Tile2D &p, int cu, int cv)
{
  const int ou = kTileWarps * cu - 2 * kTileSteps, ov = 32 * cv - 2 * kTileSteps;
  return (int64_t) ((p.nu + ou - 1) / ou) * ((p.nv + ov - 1) / ov);
}

}  // namespace

}  // namespace fdtdb
