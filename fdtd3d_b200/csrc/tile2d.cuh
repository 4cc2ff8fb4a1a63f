// tile2d.cuh - several time steps of a 2-D mode in one launch, for the FP64
// plain form (compiled with --fmad=false) and the FP32 / FP16-storage forms.
//
// A 2-D step is a chain of tiny dependent launches (E, H, two incident-grid
// steps, sources): 512^2 cells in FP32 took 24 us per step and 120 x 100 in
// FP64 21 us, all launch and L2 latency.  Here a CTA takes a tile with a halo
// of kTileSteps cells, keeps its cells' fields in registers (a warp a few rows,
// a lane a few cells of each: neighbours along a row by shuffles, across warps
// through one shared row per component) and advances up to kTileSteps steps
// with one __syncthreads per half-step; the halo's values are computed
// twice instead of exchanged, one cell of it turning invalid per step.  Every
// cell's arithmetic is the per-cell kernels', so FP64 fields keep their bits;
// FP16 storage rounds once per launch instead of once per half-step.  A run
// of 100 steps at 120 x 100 in FP64, its three fields read by the host: 2133
// -> 306 us; 200 steps at 512^2 in FP32: 4890 -> 1194 us (of which reading the
// fields is 465).
// The part of the 1-D incident grid a tile's TF/SF terms can reach advances
// in shared memory with it; a few CTAs advance the whole grid.
// FP64 keeps two levels of every field whose face cells are never updated: a
// step leaves the other level's face cells current, so a tile alternates the
// two values, and an odd number of steps per launch ends on the level that
// is written.  The level before the current one is the state a launch began
// with; the last launch of a call takes one step, so that after a call it is
// the step before, as the per-cell kernels leave it.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "tile2d.h"

namespace fdtdb {

namespace {

constexpr int kTileWarps = 16;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kWindow = 192;        // incident cells a tile can reach: 66 sqrt 2 + 2 kTileSteps + margins
constexpr int kIncOwn = kTileThreads - 2 * kTileSteps;

__device__ __forceinline__ double tile_ld (const double *p, int64_t i) { return p[i]; }
__device__ __forceinline__ float tile_ld (const float *p, int64_t i) { return p[i]; }
__device__ __forceinline__ float tile_ld (const __half *p, int64_t i) { return __half2float (p[i]); }
__device__ __forceinline__ void tile_st (double *p, int64_t i, double v) { p[i] = v; }
__device__ __forceinline__ void tile_st (float *p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void tile_st (__half *p, int64_t i, float v) { p[i] = __float2half_rn (v); }

// N neighbouring shared values (a lane's cells of a row: one 8-byte access for
// two floats, where two scalar ones would each hit every bank twice).
template <int N, typename C>
__device__ __forceinline__ void lds_row (const C *p, C v[N])
{
  if constexpr (N == 2 && sizeof (C) == 4)
  {
    const float2 t = *reinterpret_cast<const float2 *> (p);
    v[0] = t.x;
    v[1] = t.y;
  }
  else
#pragma unroll
    for (int i = 0; i < N; ++i)
      v[i] = p[i];
}
template <int N, typename C>
__device__ __forceinline__ void sts_row (C *p, const C v[N])
{
  if constexpr (N == 2 && sizeof (C) == 4)
    *reinterpret_cast<float2 *> (p) = make_float2 (v[0], v[1]);
  else
#pragma unroll
    for (int i = 0; i < N; ++i)
      p[i] = v[i];
}

// The incident grid on [c0, c0 + n) in shared memory: E, then H step.  Cells
// whose neighbour lies outside the window turn invalid from its ends inwards.
// (Rounded operations: the same bits in every form.)
__device__ __forceinline__ void inc_e_step (double *e, const double *h, int c0, int n, const Tile2D &p, double src)
{
  const int q = threadIdx.x + 32 * threadIdx.y, i = c0 + q;
  if (q < n && i < p.inc_len)
  {
    if (i == 0)
      e[q] = src;
    else if (q > 0)
      e[q] = __dadd_rn (e[q], __dmul_rn (__dsub_rn (h[q - 1], h[q]), p.mod_e));
  }
}
__device__ __forceinline__ void inc_h_step (double *h, const double *e, int c0, int n, const Tile2D &p)
{
  const int q = threadIdx.x + 32 * threadIdx.y, i = c0 + q;
  if (q + 1 < n && i < p.inc_len - 1)
    h[q] = __dadd_rn (h[q], __dmul_rn (__dsub_rn (e[q], e[q + 1]), p.mod_h));
}

// One border term of a cell, resolved once per launch: the two incident cells
// it interpolates (window index q, weight pr2 of the second), its projection
// with sign, and the neighbour (slot) of the curl it corrects.
struct TileTerm
{
  int q, slot;
  double pr2, proj;
};

// The term's place in the window for component k at cell (u, v) (the
// expressions of the per-cell kernels' incident value).
__device__ __noinline__ TileTerm tile_term (const Tile2D *p, const TermDev *tm, int c0, int u, int v)
{
  const int k = tm->inc_comp;
  const double du = ((double) (u + tm->aux[0]) + p->pos[k][0]) - p->zero[0];
  const double dv = ((double) (v + tm->aux[1]) + p->pos[k][1]) - p->zero[1];
  const double d = du * p->k[0] + dv * p->k[1] - (k >= 3 ? 0.5 : 0.0);
  const double cd1 = (double) ((int) d);
  TileTerm t;
  t.pr2 = d - cd1;
  t.q = (int) cd1 - c0;
  t.slot = tm->slot;
  t.proj = p->proj[k] * tm->negate;
  if ((int) cd1 < 0 || (int) cd1 + 1 >= p->inc_len || t.q < 0 || t.q + 1 >= kWindow)
  {
    *p->err = 1;
    t.q = 0;
    t.proj = 0.0;
  }
  return t;
}

// E-from-D's two coefficients (out of line: four IEEE divisions).
__device__ __noinline__ double2 tile_coeffs (double plus, double minus, double modifier, double dd)
{
  const double a = (plus / modifier) / dd;
  return make_double2 (a, minus == plus ? a : (minus / modifier) / dd);
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

// Shared memory of a tile, in values of the arithmetic type: the rows that
// warps exchange (one per component and warp), per-cell coefficients (FP64:
// E-from-D's two, or without PML the curl's; FP32: S / m, in PML cells 1 / m)
// and the 1-D PML tables along the tile; then the border terms.
template <typename C, int RU, int RV>
struct TileMem
{
  static constexpr int TU = kTileWarps * RU, TV = 32 * RV, TM = TU > TV ? TU : TV, N = TU * TV;
  static constexpr int ROWS = 3 * kTileWarps * TV;
  static constexpr int COEF = ROWS, TAB = COEF + (sizeof (C) == 8 ? 6 : 3) * N;
  static constexpr int TERMS = 8 * TM;   // at most eight border lines cross a tile
  static constexpr int TERM_OFF = (TAB + 3 * 6 * TM) * (int) sizeof (C);
  static constexpr int BYTES = TERM_OFF + TERMS * (int) sizeof (TileTerm);
};

// T: stored field type, C: arithmetic (double or float).  Warp w holds the RU
// rows u0 + RU w ..., a lane RV neighbouring cells of each: differences along
// v cross lanes by shuffles, those along u cross warps by one shared row per
// component, all others stay in the thread's registers.
// CHAIN: the coefficients, tables and border terms are set up before the launch
// in front of this one is over, the fields loaded after it.
template <typename T, typename C, int RU, int RV, int FORM, bool CHAIN>
__device__ __forceinline__ void tile2d_steps (const Tile2D &p, int u0, int v0, unsigned char *smem,
                                              double (*s_inc)[kTileThreads])
{
  constexpr bool F64 = sizeof (C) == 8;
  using L = TileMem<C, RU, RV>;
  using M = Mode2D<FORM>;
  constexpr int TU = L::TU, TV = L::TV, TM = L::TM, N = L::N, R = RU * RV;
  constexpr unsigned kAll = 0xffffffffu;
  C *const Row = reinterpret_cast<C *> (smem), *const K = Row + L::COEF, *const Tab = Row + L::TAB;
  TileTerm *const Terms = reinterpret_cast<TileTerm *> (smem + L::TERM_OFF);
  __shared__ int s_terms;
  const int lane = threadIdx.x, w = threadIdx.y;
  const int row0 = RU * w, col0 = RV * lane;
  const int ub = u0 + row0, vb = v0 + col0;
  if (lane + 32 * w == 0)
    s_terms = 0;

  if (p.use_pml)
    for (int q = lane + 32 * w; q < 3 * 6 * TM; q += kTileThreads)
    {
      const int j = q / (6 * TM), t = (q / TM) % 6, i = q % TM;
      const TileComp &c = p.comp[j];
      const int ax = t < 2 ? M::ax1 (j) : (t < 4 ? M::ax5 (j) : M::ax4 (j));
      const int g = ax == 0 ? u0 + i : (ax == 1 ? v0 + i : 0), n = ax == 0 ? p.nu : (ax == 1 ? p.nv : 1);
      Tab[q] = g >= 0 && g < n ? ((const C *) c.tab[t])[g] : C (1);
    }

  // ---- this thread's cells (bit RV r + c of the masks): field and PML
  // auxiliary.  (FP64 face cells keep the other level's field in the
  // auxiliary's place, which they do not have.)  Every load of a kind is
  // issued before any is used.
  C f[3][RU][RV], x[3][RU][RV];
  unsigned upd = 0, face = 0, source = 0, in_pml[3] = {0, 0, 0};
  int64_t ids[RU];
  auto load = [&] (int j, int r, int c, bool valid, bool up, bool pm) __attribute__ ((always_inline)) {
    const TileComp &q = p.comp[j];
    f[j][r][c] = C (0);
    x[j][r][c] = C (0);
    if (valid)
      f[j][r][c] = C (tile_ld ((const T *) q.in, ids[r] + c));
    if constexpr (F64)
    {
      const C *const src = !up ? (const C *) q.out : (const C *) q.aux_in;
      if (valid && src)
        x[j][r][c] = src[ids[r] + c];
    }
    else if (pm)
      x[j][r][c] = ((const float *) q.aux_in)[ids[r] + c];
  };
#pragma unroll
  for (int r = 0; r < RU; ++r)
  {
    const int u = ub + r;
    const bool uv = u >= 0 && u < p.nu, uu = u >= 1 && u <= p.nu - 2;
    ids[r] = (int64_t) (uv ? u : 0) * p.nv + vb;
#pragma unroll
    for (int c = 0; c < RV; ++c)
    {
      const int v = vb + c;
      const unsigned bit = 1u << (RV * r + c);
      const bool valid = uv && v >= 0 && v < p.nv, up = uu && v >= 1 && v <= p.nv - 2;
      upd |= up ? bit : 0u;
      face |= valid && !up ? bit : 0u;
      source |= up && u == p.pu && v == p.pv ? bit : 0u;
#pragma unroll
      for (int j = 0; j < 3; ++j)
      {
        const TileComp &q = p.comp[j];
        const bool pm =
            !F64 && up && p.use_pml && !(u >= q.ilo[0] && u < q.ihi[0] && v >= q.ilo[1] && v < q.ihi[1]);
        if constexpr (!CHAIN)
          load (j, r, c, valid, up, pm);
        in_pml[j] |= pm ? bit : 0u;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
  {
    const TileComp &q = p.comp[j];
    C m[RU][RV];
#pragma unroll
    for (int r = 0; r < RU; ++r)
#pragma unroll
      for (int c = 0; c < RV; ++c)
        m[r][c] = C (1);
    if (q.mat)
    {
      const C *const mat = (const C *) q.mat;
      const int o1 = q.m[1][0] * p.nv + q.m[1][1], o2 = q.m[2][0] * p.nv + q.m[2][1], o3 = q.m[3][0] * p.nv + q.m[3][1];
#pragma unroll
      for (int r = 0; r < RU; ++r)
#pragma unroll
        for (int c = 0; c < RV; ++c)
          if ((upd >> (RV * r + c)) & 1u)
          {
            const int64_t id = ids[r] + c;
            const C a = mat[id], b = q.nmat > 1 ? mat[id + o1] : C (0);
            const C d = q.nmat > 2 ? mat[id + o2] : C (0), e = q.nmat > 2 ? mat[id + o3] : C (0);
            if constexpr (F64)
              m[r][c] = q.nmat == 1 ? a : (q.nmat == 2 ? (a + b) / 2.0 : ((a + b) / 2.0 + (d + e) / 2.0) / 2.0);
            else
              m[r][c] = q.nmat == 1 ? a : (q.nmat == 2 ? 0.5f * (a + b) : 0.25f * (a + b + d + e));
          }
    }
    else if (!F64)
      continue;   // (FP32 without a map: S, or 1 in PML cells, is not read from K)
#pragma unroll
    for (int r = 0; r < RU; ++r)
#pragma unroll
      for (int c = 0; c < RV; ++c)
        if ((upd >> (RV * r + c)) & 1u)
        {
          const int u = ub + r, v = vb + c, at = j * N + (row0 + r) * TV + col0 + c;
          if constexpr (F64)
          {
            const double mm = p.mm[M::is_h (j)];
            if (p.use_pml)
            {
              const C *const *tab = (const C *const *) q.tab;
              const int q5 = M::ax5 (j) == 0 ? u : (M::ax5 (j) == 1 ? v : 0);
              const int q4 = M::ax4 (j) == 0 ? u : (M::ax4 (j) == 1 ? v : 0);
              const double2 k = tile_coeffs (tab[4][q4], tab[5][q4], m[r][c] * mm, tab[3][q5]);
              K[at] = k.x;
              K[3 * N + at] = k.y;
            }
            else
              K[at] = p.dt / (m[r][c] * mm * p.dx);
          }
          else
            K[at] = (in_pml[j] >> (RV * r + c)) & 1u ? 1.f / m[r][c] : p.courant * (1.f / m[r][c]);
        }
  }
  // border terms of the tile: first how many (a tile without any has none of
  // the incident grid's work), then their window and their entries, E's and
  // H's of a thread one after the other in the order the half-steps take them
  unsigned terms[(R + 1) / 2] = {};   // 16 bits per cell: bit 4 j + t
  int mine = 0;
#pragma unroll
  for (int r = 0; r < RU; ++r)
#pragma unroll
    for (int c = 0; c < RV; ++c)
    {
      unsigned t12 = 0;
      if (p.use_tfsf && ((upd >> (RV * r + c)) & 1u))
#pragma unroll
        for (int j = 0; j < 3; ++j)
          for (int t = 0; t < p.comp[j].nterms; ++t)
          {
            const TermDev &tm = p.comp[j].term[t];
            if (ub + r >= tm.lo[0] && ub + r < tm.hi[0] && vb + c >= tm.lo[1] && vb + c < tm.hi[1])
              t12 |= 1u << (4 * j + t);
          }
      terms[(RV * r + c) / 2] |= t12 << (16 * ((RV * r + c) & 1));
      mine += __popc (t12);
    }
  const bool has_terms = __syncthreads_or (mine) != 0;
  int wc = 0, first[2] = {0, 0};
  auto window = [&] () __attribute__ ((always_inline)) {
    const int q = lane + 32 * w, i = wc + q;
    if (q < kWindow)
    {
      s_inc[0][q] = i < p.inc_len ? p.e_in[i] : 0.0;
      s_inc[1][q] = i < p.inc_len ? p.h_in[i] : 0.0;
    }
  };
  if (has_terms)
  {
    const double a0 = ((double) (u0 - 1) - p.zero[0]) * p.k[0], a1 = ((double) (u0 + TU + 1) - p.zero[0]) * p.k[0];
    const double b0 = ((double) (v0 - 1) - p.zero[1]) * p.k[1], b1 = ((double) (v0 + TV + 1) - p.zero[1]) * p.k[1];
    wc = max (0, (int) (fmin (a0, a1) + fmin (b0, b1)) - kTileSteps - 3);
    if constexpr (!CHAIN)
      window ();
    if (mine)
    {
      int e = atomicAdd (&s_terms, mine);
#pragma unroll
      for (int fam = 0; fam < 2; ++fam)
      {
        first[fam] = e;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (M::is_h (j) == (fam == 1))
#pragma unroll
            for (int r = 0; r < RU; ++r)
#pragma unroll
              for (int c = 0; c < RV; ++c)
                for (unsigned t = (terms[(RV * r + c) / 2] >> (16 * ((RV * r + c) & 1) + 4 * j)) & 15u; t; t &= t - 1, ++e)
                  if (e < L::TERMS)
                    Terms[e] = tile_term (&p, &p.comp[j].term[__ffs ((int) t) - 1], wc, ub + r, vb + c);
      }
    }
  }

  // (all above reads only what no step writes)
  if constexpr (CHAIN)
  {
    cudaGridDependencySynchronize ();
    if (has_terms)
      window ();
#pragma unroll
    for (int r = 0; r < RU; ++r)
#pragma unroll
      for (int c = 0; c < RV; ++c)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          load (j, r, c, ((upd | face) >> (RV * r + c)) & 1u, (upd >> (RV * r + c)) & 1u,
                (in_pml[j] >> (RV * r + c)) & 1u);
  }

  // the row a neighbouring warp reads of component j: the last one where the
  // other family looks down (u - 1), the first where it looks up
  auto publish = [&] (auto j_c) __attribute__ ((always_inline)) {
    constexpr int j = decltype (j_c)::value;
    // (a component of the other family: E is the first one, H the last)
    constexpr int r = M::low (M::is_h (j) ? 0 : 2) == -1 ? RU - 1 : 0;
    sts_row<RV> (Row + (j * kTileWarps + w) * TV + col0, f[j][r]);
  };
  publish (std::integral_constant<int, 0>{});
  publish (std::integral_constant<int, 1>{});
  publish (std::integral_constant<int, 2>{});
  __syncthreads ();

  // whether this warp's cells need border terms or the source
  const bool rare = __any_sync (kAll, mine != 0 || source != 0);
  const C plain_kc = C (p.courant);   // FP32 cells without a material map

  // One half-step of the family FAM.
  auto half = [&] (auto fam_c, auto rare_c, int s) __attribute__ ((always_inline)) {
    constexpr int FAM = decltype (fam_c)::value;
    constexpr bool RARE = decltype (rare_c)::value;
    int entry = first[FAM];
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
      const TileComp &q = p.comp[j];
      if (M::is_h (j) != (FAM == 1))
        continue;
      // far neighbours of the two differences (0 where one is absent)
      C far[2][RU][RV];
#pragma unroll
      for (int i = 0; i < 2; ++i)
      {
        const int sl = M::opp (j, i) < 0 ? 0 : M::opp (j, i);
        const bool down = M::low (j) == -1;
#pragma unroll
        for (int r = 0; r < RU; ++r)
#pragma unroll
          for (int c = 0; c < RV; ++c)
            far[i][r][c] = C (0);
        if (M::opp (j, i) < 0)
          continue;
        if (M::along (j, i) == 0)
        {
          const int nb = down ? max (w - 1, 0) : min (w + 1, kTileWarps - 1);
          C other[RV];
          lds_row<RV> (Row + (sl * kTileWarps + nb) * TV + col0, other);
#pragma unroll
          for (int r = 0; r < RU; ++r)
#pragma unroll
            for (int c = 0; c < RV; ++c)
              far[i][r][c] = down ? (r > 0 ? f[sl][r > 0 ? r - 1 : 0][c] : other[c])
                                  : (r < RU - 1 ? f[sl][r < RU - 1 ? r + 1 : 0][c] : other[c]);
        }
        else
        {
#pragma unroll
          for (int r = 0; r < RU; ++r)
          {
            const C other = down ? __shfl_up_sync (kAll, f[sl][r][RV - 1], 1) : __shfl_down_sync (kAll, f[sl][r][0], 1);
#pragma unroll
            for (int c = 0; c < RV; ++c)
              far[i][r][c] = down ? (c > 0 ? f[sl][r][c > 0 ? c - 1 : 0] : other)
                                  : (c < RV - 1 ? f[sl][r][c < RV - 1 ? c + 1 : 0] : other);
          }
        }
      }
      // the curls, border terms subtracted from their neighbours
      C cu[RU][RV];
#pragma unroll
      for (int r = 0; r < RU; ++r)
#pragma unroll
        for (int c = 0; c < RV; ++c)
        {
          const int bit = RV * r + c;
          const bool down = M::low (j) == -1;
          const int s1 = M::opp (j, 0), s2 = M::opp (j, 1);
          const C n1 = s1 < 0 ? C (0) : f[s1 < 0 ? 0 : s1][r][c], n2 = s2 < 0 ? C (0) : f[s2 < 0 ? 0 : s2][r][c];
          C a = down ? far[0][r][c] : n1, b = down ? n1 : far[0][r][c];
          C d = down ? far[1][r][c] : n2, e = down ? n2 : far[1][r][c];
          if (RARE)
            for (unsigned t = (terms[bit / 2] >> (16 * (bit & 1) + 4 * j)) & 15u; t; t &= t - 1, ++entry)
            {
              const TileTerm y = Terms[entry];
              const double *const win = s_inc[FAM == 0 ? 1 : 0];   // (the terms are of the other family)
              const double v = (win[y.q] * (1 - y.pr2) + win[y.q + 1] * y.pr2) * y.proj;
              const C z = F64 ? C (v) : C ((float) v * p.scale[FAM == 0 ? 1 : 0]);
              a = y.slot == 0 ? a - z : a;
              b = y.slot == 1 ? b - z : b;
              d = y.slot == 2 ? d - z : d;
              e = y.slot == 3 ? e - z : e;
            }
          cu[r][c] = F64 ? b - a - e + d : (b - a) - (e - d);
        }
      if constexpr (F64)
      {
        const C *const t = Tab + 6 * j * TM;
#pragma unroll
        for (int r = 0; r < RU; ++r)
#pragma unroll
          for (int c = 0; c < RV; ++c)
          {
            const int bit = RV * r + c, ak = j * N + (row0 + r) * TV + col0 + c;
            const int q1 = M::ax1 (j) == 0 ? row0 + r : (M::ax1 (j) == 1 ? col0 + c : 0);
            const int q5 = M::ax5 (j) == 0 ? row0 + r : (M::ax5 (j) == 1 ? col0 + c : 0);
            const C of = f[j][r][c], ox = x[j][r][c], kc = K[ak];
            C nf, nx = ox;
            if (p.use_pml)
            {
              nx = ox * t[q1] + cu[r][c] * t[TM + q1];
              nf = of * t[2 * TM + q5] + nx * kc - ox * K[3 * N + ak];
            }
            else
              nf = of + cu[r][c] * kc;
            // (a face cell alternates with the other level's value)
            const bool up = (upd >> bit) & 1u, fc = (face >> bit) & 1u;
            f[j][r][c] = up ? nf : (fc ? ox : of);
            x[j][r][c] = up ? nx : (fc ? of : ox);
          }
      }
      else if (!__any_sync (kAll, in_pml[j]))
      {
        const bool has_k = q.mat != nullptr;
#pragma unroll
        for (int r = 0; r < RU; ++r)
        {
          C kv[RV];
          if (has_k)
            lds_row<RV> (K + j * N + (row0 + r) * TV + col0, kv);
#pragma unroll
          for (int c = 0; c < RV; ++c)
          {
            const C nf = f[j][r][c] + (has_k ? kv[c] : plain_kc) * cu[r][c];
            f[j][r][c] = (upd >> (RV * r + c)) & 1u ? nf : f[j][r][c];
          }
        }
      }
      else
      {
        // the component's PML values along its axes: one set per row, per
        // column, or one
        constexpr int NT = RU > RV ? RU : RV;
        C tb[6][NT];
#pragma unroll
        for (int t = 0; t < 6; ++t)
        {
          const int ax = t < 2 ? M::ax1 (j) : (t < 4 ? M::ax5 (j) : M::ax4 (j));
          const C *const from = Tab + (6 * j + t) * TM + (ax == 0 ? row0 : (ax == 1 ? col0 : 0));
#pragma unroll
          for (int i = 0; i < (ax == 0 ? RU : (ax == 1 ? RV : 1)); ++i)
            tb[t][i] = from[i];
        }
        const bool has_k = q.mat != nullptr;
#pragma unroll
        for (int r = 0; r < RU; ++r)
        {
          C kv[RV];
          if (has_k)
            lds_row<RV> (K + j * N + (row0 + r) * TV + col0, kv);
#pragma unroll
          for (int c = 0; c < RV; ++c)
          {
            const int bit = RV * r + c;
            const int i1 = M::ax1 (j) == 0 ? r : (M::ax1 (j) == 1 ? c : 0);
            const int i5 = M::ax5 (j) == 0 ? r : (M::ax5 (j) == 1 ? c : 0);
            const int i4 = M::ax4 (j) == 0 ? r : (M::ax4 (j) == 1 ? c : 0);
            const bool pm = (in_pml[j] >> bit) & 1u, up = (upd >> bit) & 1u;
            const C of = f[j][r][c], ox = x[j][r][c];
            const C nf = of + (has_k ? kv[c] : plain_kc) * cu[r][c];
            const C nx = tb[0][i1] * ox + tb[1][i1] * cu[r][c];
            const C pf = tb[2][i5] * of + (tb[4][i4] * nx - tb[5][i4] * ox) * tb[3][i5] * (has_k ? kv[c] : C (1));
            f[j][r][c] = pm ? pf : (up ? nf : of);
            x[j][r][c] = pm ? nx : ox;
          }
        }
      }
      if (RARE && q.source && source)
      {
#pragma unroll
        for (int r = 0; r < RU; ++r)
#pragma unroll
          for (int c = 0; c < RV; ++c)
            if ((source >> (RV * r + c)) & 1u)
              f[j][r][c] =
                  F64 ? C (p.src[p.src_row * s + 1 + FAM]) : C ((float) p.src[p.src_row * s + 1 + FAM] * p.scale[FAM]);
      }
    }
    // (both components of a family are updated from the other family only,
    // so the rows are published after all of them)
    if (M::is_h (0) == (FAM == 1))
      publish (std::integral_constant<int, 0>{});
    if (M::is_h (1) == (FAM == 1))
      publish (std::integral_constant<int, 1>{});
    if (M::is_h (2) == (FAM == 1))
      publish (std::integral_constant<int, 2>{});
  };
  auto any_half = [&] (auto fam_c, int s) __attribute__ ((always_inline)) {
    if (!rare)
      half (fam_c, std::false_type{}, s);
    else
      half (fam_c, std::true_type{}, s);
  };
#pragma unroll 1
  for (int s = 0; s < p.steps; ++s)
  {
    // the incident grid's half-step touches the family the terms do not
    // read: E terms read HInc before its update, H terms EInc after its
    if (has_terms)
      inc_e_step (s_inc[0], s_inc[1], wc, kWindow, p, p.src[p.src_row * s]);
    any_half (std::integral_constant<int, 0>{}, s);
    __syncthreads ();
    if (has_terms)
      inc_h_step (s_inc[1], s_inc[0], wc, kWindow, p);
    any_half (std::integral_constant<int, 1>{}, s);
    __syncthreads ();
  }

#pragma unroll
  for (int r = 0; r < RU; ++r)
#pragma unroll
    for (int c = 0; c < RV; ++c)
    {
      const int du = row0 + r, dv = col0 + c, bit = RV * r + c;
      if (!((upd >> bit) & 1u) || du < kTileSteps || du >= TU - kTileSteps || dv < kTileSteps || dv >= TV - kTileSteps)
        continue;
#pragma unroll
      for (int j = 0; j < 3; ++j)
      {
        tile_st ((T *) p.comp[j].out, ids[r] + c, f[j][r][c]);
        if (p.use_pml && (F64 || ((in_pml[j] >> bit) & 1u)))
          ((C *) p.comp[j].aux_out)[ids[r] + c] = x[j][r][c];
      }
    }
}

template <typename T, typename C, int RU, int RV, int FORM>
__global__ void __launch_bounds__ (kTileThreads, 1) tile2d_kernel (const __grid_constant__ Tile2D p, int tiles_v,
                                                                  int ntiles)
{
  constexpr int OU = kTileWarps * RU - 2 * kTileSteps, OV = 32 * RV - 2 * kTileSteps;
  extern __shared__ __align__ (16) unsigned char tile_smem[];
  __shared__ double s_inc[2][kTileThreads];
  // The next launch may begin while this one steps: its launch latency, and on
  // the SMs that small tiles leave free its set-up, are then not in the chain.
  // Seven steps: 120 x 100 with TF/SF FP64 24.7 -> 16.2 us, FP32 21.8 -> 14.6;
  // 200 x 200 FP32 13.3 -> 9.6.  (Tiles of more cells fill the SMs' registers,
  // so nothing of the next launch runs before this one ends: with the late
  // loads they spill and 512 x 512 FP32 takes 27.9 us instead of 26.6.)
  constexpr bool CHAIN = RU * RV == 2;
  cudaTriggerProgrammaticLaunchCompletion ();
  if (!CHAIN || (int) blockIdx.x >= ntiles)
    cudaGridDependencySynchronize ();
  if ((int) blockIdx.x >= ntiles)
  {
    const int lane = threadIdx.x, w = threadIdx.y;
    // a stretch of the incident grid
    const int c0 = ((int) blockIdx.x - ntiles) * kIncOwn - kTileSteps, q = lane + 32 * w, i = c0 + q;
    const bool in = i >= 0 && i < p.inc_len;
    s_inc[0][q] = in ? p.e_in[i] : 0.0;
    s_inc[1][q] = in ? p.h_in[i] : 0.0;
    __syncthreads ();
    for (int s = 0; s < p.steps; ++s)
    {
      if (i >= 0)
        inc_e_step (s_inc[0], s_inc[1], c0, kTileThreads, p, p.src[p.src_row * s]);
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
  tile2d_steps<T, C, RU, RV, FORM, CHAIN> (p, ((int) blockIdx.x / tiles_v) * OU - kTileSteps,
                                    ((int) blockIdx.x % tiles_v) * OV - kTileSteps, tile_smem, s_inc);
}

template <typename T, typename C, int RU, int RV, int FORM>
int tile2d_start (const Tile2D &p, cudaStream_t s)
{
  constexpr int OU = kTileWarps * RU - 2 * kTileSteps, OV = 32 * RV - 2 * kTileSteps;
  constexpr int smem = TileMem<C, RU, RV>::BYTES;
  const int tu = (p.nu + OU - 1) / OU, tv = (p.nv + OV - 1) / OV;
  const int inc = p.use_tfsf ? (p.inc_cells + kIncOwn - 1) / kIncOwn : 0;
  auto kern = tile2d_kernel<T, C, RU, RV, FORM>;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3 (tu * tv + inc);
  lc.blockDim = dim3 (32, kTileWarps);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = &at;
  lc.numAttrs = 1;
  cudaLaunchKernelEx (&lc, kern, p, tv, tu * tv);
  return 1;
}

template <typename T, typename C, int RU, int RV>
int tile2d_launch (const Tile2D &p, cudaStream_t s)
{
  switch ((p.form.te ? 1 : 0) + (p.form.flip ? 2 : 0) + (p.form.hc ? 4 : 0))
  {
    case 0: return tile2d_start<T, C, RU, RV, 0> (p, s);
    case 1: return tile2d_start<T, C, RU, RV, 1> (p, s);
    case 2: return tile2d_start<T, C, RU, RV, 2> (p, s);
    case 3: return tile2d_start<T, C, RU, RV, 3> (p, s);
    case 4: return tile2d_start<T, C, RU, RV, 4> (p, s);
    case 5: return tile2d_start<T, C, RU, RV, 5> (p, s);
    case 6: return tile2d_start<T, C, RU, RV, 6> (p, s);
    default: return tile2d_start<T, C, RU, RV, 7> (p, s);
  }
}

// Tiles of a launch for a tile of RU x RV cells per thread.
inline int64_t tile2d_count (const Tile2D &p, int cu, int cv)
{
  const int ou = kTileWarps * cu - 2 * kTileSteps, ov = 32 * cv - 2 * kTileSteps;
  return (int64_t) ((p.nu + ou - 1) / ou) * ((p.nv + ov - 1) / ov);
}

}  // namespace

}  // namespace fdtdb
