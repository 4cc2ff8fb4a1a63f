// adjoint.cu - checkpointed reverse-mode differentiation of the 2-D TMz
// step (see adjoint.h).
//
// Forward step k (k = 0 .. steps - 1), as the library's FP32 TMz step:
//   k > 0: Ez cells: curl of H; interior Ez += S * im * curl, PML cells
//          X_new = ca1 X + sq1 curl, Ez = p5 Ez + (g4p X_new - g4m X) q5 im
//          (im = 1 / averaged eps); Ez point source overwrites its cell;
//   k > 0: Hx, Hy the same with im = 1; H point source overwrites its cell;
//   J += sum over the probe of Ez_k^2.
// Reverse step k (k = steps - 1 .. 1), two phases:
//   H phase: aH += (curl of H)^T acz (acz stored by the E phase of step
//            k + 1), then the transpose of the H half-step of step k at each
//            H cell, storing its curl adjoints acx, acy;
//   E phase: aE += (curl of E)^T (acx, acy) + 2 Ez_k on the probe, the
//            gradient of im += aE * dEz/dim, then the transpose of the E
//            half-step of step k at each Ez cell, storing its curl adjoint acz.
// Point-source cells carry no adjoint into the step before (their value is
// overwritten).  dJ/d eps = sum over the Ez cells whose average includes
// the cell of dJ/d im * (-im^2 / n_points).
//
// Execution: one persistent cooperative kernel runs many steps in rounds of up
// to kRound with a bounded grid barrier between them.  In a round a CTA takes
// tiles of the grid with a halo of kRound cells, holds its cells in registers
// and the values neighbours read in shared memory, and recomputes the halo
// instead of exchanging it; the state is double buffered between rounds.
// (With a grid barrier per half-step the run was bound by barrier and L2
// latency, about 6 us each: 512^2, 800 steps, checkpoint 100: forward 11.3 ms,
// backward 26.3 ms; now 2.3 and 10.8 ms.)  The forward run is one launch that
// also stores the checkpoints (the state before every K-th step) and, for the
// last segment, dEz/dim and the probe values the reverse sweep needs.  Every
// reverse launch splits its CTAs in two groups with a barrier each: one group
// reverses segment j from the stored per-step data while the other recomputes
// segment j - 1 from its checkpoint into the other half of the double buffer.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "adjoint.h"
#include "kernels.h"

namespace fdtdb {

namespace {

constexpr int kEz = 0, kHx = 1, kHy = 2;   // local component slots
constexpr double kEta0Adj = 376.730313461770655;
constexpr int kThreads = 512;
constexpr int kRound = 7;                  // steps per round at most: the halo of a tile
constexpr int kBarStride = 64;             // words per group barrier: arrivals at [0], generation at [32]
constexpr long long kDefaultBarrierLimitNs = 2000000000LL;   // 2 s

template <typename R>
struct AdjDev
{
  int nx, ny;
  R S;
  int ilo[3][2], ihi[3][2];    // sigma == 0 range per component and axis
  int tax[3][3];               // axis of the (ca1, sq1), (p5, q5), (g4p, g4m) pairs
  const R *tab[3][6];          // tables indexed by the coordinate along the pair's axis
  const R *im;                 // 1 / averaged eps of Ez
  int ps[2];
  int ps_on[3];                // point source on Ez / Hx / Hy
  const R *src;                // [2k] E value, [2k + 1] H value of step k
  int pr_lo[2], pr_hi[2];
};

// One persistent launch.  CTAs [0, fwd_ctas) run forward steps fk0 .. fk1 - 1,
// the others reverse steps rk1 - 1 .. max(rk0, 1).
template <typename R>
struct Launch
{
  AdjDev<R> p;
  int N, npr;
  // forward group
  int fwd_ctas;
  uint32_t fk0, fk1;
  R *F[2];                     // two sets of Ez, Hx, Hy, Xz, Xx, Xy (N values each); a launch starts in set 0
  const R *load;               // state to start from (6 N values) instead of set 0, or null
  // state before step k stored at ck + (k / every - 1) 6 N when k % every == 0, or
  // null (not before step 0, which is 0, nor before keep0, from where the
  // per-step data are kept)
  R *ck;
  uint32_t every;
  R *dedm;                     // dEz/dim of step k at dedm + (k - keep0) N for k >= keep0, or null
  double *keep;                // probe Ez of step k at keep + (k - keep0) npr
  uint32_t keep0;
  double *jpart;               // sum of Ez^2 over the probe cells of probe tile q and all steps: a pair (sum, compensation)
                               // at 2 q, or null
  int prt_u0, prt_v0, prt_nv;  // tiles that hold probe cells
  // reverse group
  uint32_t rk0, rk1;
  R *A[2];                     // two sets of aE, aXz, aHx, aHy, aXx, aXy, acz (N values each)
  int rcur;                    // set the reverse steps start from
  const R *rdedm;              // dEz/dim of step k at rdedm + (k - rk0) N
  const double *rprobe;        // probe Ez of step k at rprobe + (k - rk0) npr
  double *gim;
  int tiles_u, tiles_v;
  // barriers: arrivals at [0] and generation at [32] for the forward group,
  // the same from [kBarStride] for the reverse group (each word in its own
  // 128-byte line, so polling does not slow the arrivals)
  unsigned *bar;
  int *err;
  long long limit_ns;          // time limit of one barrier wait
};

// values that other CTAs of the launch write are read through L2
template <typename R>
__device__ __forceinline__ R ld (const R *q)
{
  return __ldcg (q);
}

__device__ __forceinline__ long long globaltimer ()
{
  long long t;
  asm volatile ("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier over the `ctas` CTAs of one group, with a time limit.  Returns
// false (and sets *err) when any CTA gave up; every CTA then leaves.
__device__ bool group_barrier (unsigned *bar, unsigned ctas, int *err, long long limit_ns)
{
  __shared__ int ok;
  __syncthreads ();
  if (threadIdx.x == 0)
  {
    volatile unsigned *gen = bar + 32;
    const unsigned g = *gen;
    __threadfence ();
    if (atomicAdd (bar, 1u) == ctas - 1)
    {
      atomicExch (bar, 0u);
      __threadfence ();
      atomicAdd (bar + 32, 1u);
    }
    else
    {
      const long long t0 = globaltimer ();
      while (*gen == g)
      {
        if (*((volatile int *) err) != 0 || globaltimer () - t0 > limit_ns)
        {
          atomicExch (err, 1);
          break;
        }
        __nanosleep (20);
      }
    }
    __threadfence ();
    ok = *((volatile int *) err) == 0;
  }
  __syncthreads ();
  return ok != 0;
}

// Tile of 16 RU x 32 RV cells, halo included: warp w holds the RU rows u0 + RU
// w ..., a lane RV neighbouring cells of each.  Differences along y cross lanes
// by shuffles, those along x cross warps by one shared row per component.
template <typename R, int RU, int RV>
struct AdjTile
{
  static constexpr int TU = 16 * RU, TV = 32 * RV, TM = TU > TV ? TU : TV, C = RU * RV;
  static constexpr int OU = TU - 2 * kRound, OV = TV - 2 * kRound;
  static constexpr int A = 16 * TV;                    // one component's exchanged rows
  static constexpr int BYTES = (2 * A + 18 * TM) * (int) sizeof (R);
};

// What a thread knows of its cells (bit RV i + j for row i, column j): `upd`:
// an updated cell, `own`: of the tile's own part and inside the grid, `pml[c]`:
// component c has PML there.
template <typename R, int RU, int RV>
struct AdjCells
{
  using L = AdjTile<R, RU, RV>;
  int u0, v0, w, lane;
  unsigned valid = 0, upd = 0, own = 0, source = 0, pml[3] = {0, 0, 0};
  __device__ AdjCells (const AdjDev<R> &p, int u0_, int v0_) : u0 (u0_), v0 (v0_)
  {
    w = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < L::C; ++r)
    {
      const int x = u0 + du (r), y = v0 + dv (r);
      const unsigned bit = 1u << r;
      const bool in = x >= 0 && x < p.nx && y >= 0 && y < p.ny;
      const bool up = x >= 1 && x <= p.nx - 2 && y >= 1 && y <= p.ny - 2;
      valid |= in ? bit : 0u;
      upd |= up ? bit : 0u;
      own |= in && du (r) >= kRound && du (r) < L::TU - kRound && dv (r) >= kRound && dv (r) < L::TV - kRound ? bit : 0u;
      source |= up && x == p.ps[0] && y == p.ps[1] ? bit : 0u;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        pml[c] |= up && !(x >= p.ilo[c][0] && x < p.ihi[c][0] && y >= p.ilo[c][1] && y < p.ihi[c][1]) ? bit : 0u;
    }
  }
  __device__ int du (int r) const { return RU * w + r / RV; }
  __device__ int dv (int r) const { return RV * lane + r % RV; }
  __device__ int id (const AdjDev<R> &p, int r) const { return (u0 + du (r)) * p.ny + v0 + dv (r); }
};

// The PML coefficients of component c for a thread's cells, from the tile's
// tables (entry j of component c at T[(6 c + j) TM + q], q the offset along the
// pair's axis, 0 along the dropped one): ca1, sq1, p5, q5, g4p, g4m, each a
// value per row, per column or one.
template <typename R, int RU, int RV>
struct AdjCoef
{
  static constexpr int N = RU > RV ? RU : RV;
  R t[6][N];
  // Ez: x, y, z; Hx: y, z, x; Hy: z, x, y
  __device__ static constexpr int axis (int c, int pair)
  {
    return c == kEz ? pair : (c == kHx ? (pair + 1) % 3 : (pair + 2) % 3);
  }
  __device__ AdjCoef (const R *T, int TM, int c, int row, int col)
  {
#pragma unroll
    for (int j = 0; j < 6; ++j)
    {
      const int ax = axis (c, j / 2);
      const R *from = T + (6 * c + j) * TM + (ax == 0 ? row : (ax == 1 ? col : 0));
#pragma unroll
      for (int i = 0; i < (ax == 0 ? RU : (ax == 1 ? RV : 1)); ++i)
        t[j][i] = from[i];
    }
  }
  __device__ R at (int c, int j, int r) const
  {
    const int ax = axis (c, j / 2);
    return t[j][ax == 0 ? r / RV : (ax == 1 ? r % RV : 0)];
  }
};

// Shared PML tables of a tile.
template <typename R, int RU, int RV>
__device__ __forceinline__ void adj_tables (const AdjDev<R> &p, R *T, int u0, int v0)
{
  using L = AdjTile<R, RU, RV>;
  for (int q = threadIdx.x; q < 18 * L::TM; q += kThreads)
  {
    const int c = q / (6 * L::TM), j = (q / L::TM) % 6, i = q % L::TM;
    const int ax = p.tax[c][j / 2];
    const int g = ax == 0 ? u0 + i : (ax == 1 ? v0 + i : 0), n = ax == 0 ? p.nx : (ax == 1 ? p.ny : 1);
    T[q] = g >= 0 && g < n ? p.tab[c][j][g] : R (1);
  }
}

// A thread's row r of component f as its neighbours see it: the value one
// cell lower (D = -1) or higher (D = +1) in y, and the row of the warp before
// or after in x (row: the warps' exchanged rows).
template <typename R, int RU, int RV, int D>
__device__ __forceinline__ void adj_far_y (const R f[RU * RV], R far[RU * RV])
{
#pragma unroll
  for (int i = 0; i < RU; ++i)
  {
    const R o = D < 0 ? __shfl_up_sync (0xffffffffu, f[RV * i + RV - 1], 1) : __shfl_down_sync (0xffffffffu, f[RV * i], 1);
#pragma unroll
    for (int j = 0; j < RV; ++j)
      far[RV * i + j] = D < 0 ? (j > 0 ? f[RV * i + (j > 0 ? j - 1 : 0)] : o)
                              : (j < RV - 1 ? f[RV * i + (j < RV - 1 ? j + 1 : 0)] : o);
  }
}
template <typename R, int RU, int RV, int D>
__device__ __forceinline__ void adj_far_x (const R f[RU * RV], R far[RU * RV], const R *row, int w, int lane)
{
  const int nb = D < 0 ? max (w - 1, 0) : min (w + 1, 15);
#pragma unroll
  for (int j = 0; j < RV; ++j)
  {
    const R o = row[nb * 32 * RV + RV * lane + j];
#pragma unroll
    for (int i = 0; i < RU; ++i)
      far[RV * i + j] = D < 0 ? (i > 0 ? f[RV * (i > 0 ? i - 1 : 0) + j] : o)
                              : (i < RU - 1 ? f[RV * (i < RU - 1 ? i + 1 : 0) + j] : o);
  }
}
// The row the warp next to this one reads: the last where it looks down, the
// first where it looks up.
template <typename R, int RU, int RV, int D>
__device__ __forceinline__ void adj_publish (const R f[RU * RV], R *row, int w, int lane)
{
#pragma unroll
  for (int j = 0; j < RV; ++j)
    row[w * 32 * RV + RV * lane + j] = f[RV * (D < 0 ? RU - 1 : 0) + j];
}

// ---- forward group

// Component c's update on a thread's cells given their curls; d gets dF/d(im).
template <typename R, int RU, int RV>
__device__ __forceinline__ void adj_update (const R *T, int c, const AdjCells<R, RU, RV> &cells, R S,
                                            const R cu[RU * RV], const R *im, R f[RU * RV], R x[RU * RV], R d[RU * RV])
{
  using G = AdjTile<R, RU, RV>;
  if (!__any_sync (0xffffffffu, cells.pml[c]))
  {
#pragma unroll
    for (int r = 0; r < G::C; ++r)
    {
      d[r] = S * cu[r];
      f[r] = (cells.upd >> r) & 1u ? f[r] + S * (im ? im[r] : R (1)) * cu[r] : f[r];
    }
    return;
  }
  const AdjCoef<R, RU, RV> k (T, G::TM, c, RU * cells.w, RV * cells.lane);
#pragma unroll
  for (int r = 0; r < G::C; ++r)
  {
    const R m = im ? im[r] : R (1);
    const R xn = k.at (c, 0, r) * x[r] + k.at (c, 1, r) * cu[r];
    const R pd = (k.at (c, 4, r) * xn - k.at (c, 5, r) * x[r]) * k.at (c, 3, r);
    const R pf = k.at (c, 2, r) * f[r] + pd * m, nf = f[r] + S * m * cu[r];
    const bool pm = (cells.pml[c] >> r) & 1u, up = (cells.upd >> r) & 1u;
    d[r] = pm ? pd : S * cu[r];
    f[r] = pm ? pf : (up ? nf : f[r]);
    x[r] = pm ? xn : x[r];
  }
}

// (s, c) += v, the rounding error of the sum kept in c.
__device__ __forceinline__ void adj_add (double &s, double &c, double v)
{
  const double t = s + v, z = t - s;
  c += (s - (t - z)) + (v - z);
  s = t;
}

// Steps k0 .. k0 + steps - 1 of one tile, from `in` to `out`.
template <typename R, int RU, int RV>
__device__ void forward_tile (const Launch<R> &L, const R *in, R *out, int tu, int tv, uint32_t k0, int steps, R *S,
                              double *s_sum)
{
  using G = AdjTile<R, RU, RV>;
  const AdjDev<R> &p = L.p;
  const size_t N = L.N;
  const int u0 = tu * G::OU - kRound, v0 = tv * G::OV - kRound;
  R *const ERow = S, *const HRow = S + G::A, *const T = S + 2 * G::A;
  const AdjCells<R, RU, RV> c (p, u0, v0);
  R f[3][G::C], x[3][G::C], im[G::C];
#pragma unroll
  for (int r = 0; r < G::C; ++r)
  {
    const bool v = (c.valid >> r) & 1u;
    const int id = v ? c.id (p, r) : 0;
#pragma unroll
    for (int q = 0; q < 3; ++q)
    {
      f[q][r] = v ? ld (in + q * N + id) : R (0);
      x[q][r] = (c.pml[q] >> r) & 1u ? ld (in + (3 + q) * N + id) : R (0);
    }
    im[r] = (c.upd >> r) & 1u ? p.im[id] : R (0);
  }
  adj_tables<R, RU, RV> (p, T, u0, v0);
  if (L.ck && k0 % L.every == 0 && k0 > 0 && k0 < L.keep0)
  {
    R *const save = L.ck + (size_t) (k0 / L.every - 1) * 6 * N;
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      if ((c.own >> r) & 1u)
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
          save[q * N + c.id (p, r)] = f[q][r];
          save[(3 + q) * N + c.id (p, r)] = x[q][r];
        }
  }
  const bool probe = u0 + kRound < p.pr_hi[0] && u0 + kRound + G::OU > p.pr_lo[0] && v0 + kRound < p.pr_hi[1] &&
                     v0 + kRound + G::OV > p.pr_lo[1];
  // the tile's sum so far, thread 0's (the same CTA takes a tile in every round,
  // and the steps are added one by one: how they fall into rounds changes nothing)
  auto j_at = [&] { return L.jpart + 2 * ((size_t) (tu - L.prt_u0) * L.prt_nv + (tv - L.prt_v0)); };
  if (probe && L.jpart && threadIdx.x < 2)
    s_sum[kThreads / 32 + threadIdx.x] = j_at ()[threadIdx.x];
  // Ez reads Hy one row lower, Hy reads Ez one row higher
  adj_publish<R, RU, RV, -1> (f[2], HRow, c.w, c.lane);
  __syncthreads ();
#pragma unroll 1
  for (int s = 0; s < steps; ++s)
  {
    const uint32_t k = k0 + s;
    const bool kept = L.dedm && k >= L.keep0;
    R *const dd = kept ? L.dedm + (size_t) (k - L.keep0) * N : nullptr;
    double sum = 0.0;
    R cu[G::C], d[G::C];
    if (k > 0)
    {
      R a[G::C], b[G::C];
      adj_far_x<R, RU, RV, -1> (f[2], a, HRow, c.w, c.lane);
      adj_far_y<R, RU, RV, -1> (f[1], b);
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        cu[r] = (f[2][r] - a[r]) - (f[1][r] - b[r]);
      adj_update<R, RU, RV> (T, kEz, c, p.S, cu, im, f[0], x[0], d);
    }
    else
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        d[r] = 0;
    }
    if (p.ps_on[kEz] && c.source)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((c.source >> r) & 1u)
          f[0][r] = p.src[2 * k];
    }
    if (dd)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((c.own & c.upd) >> r & 1u)
          dd[c.id (p, r)] = d[r];
    }
    if (probe)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
      {
        const int a = u0 + c.du (r) - p.pr_lo[0], b = v0 + c.dv (r) - p.pr_lo[1], n = p.pr_hi[1] - p.pr_lo[1];
        if (((c.own & c.upd) >> r & 1u) && a >= 0 && a < p.pr_hi[0] - p.pr_lo[0] && b >= 0 && b < n)
        {
          const double v = (double) f[0][r];
          sum += v * v;
          if (kept)
            L.keep[(size_t) (k - L.keep0) * L.npr + a * n + b] = v;
        }
      }
    }
    adj_publish<R, RU, RV, 1> (f[0], ERow, c.w, c.lane);
    __syncthreads ();
    if (probe && L.jpart)
    {
      for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync (0xffffffffu, sum, o);
      if (c.lane == 0)
        s_sum[c.w] = sum;
    }
    if (k > 0)
    {
      adj_far_y<R, RU, RV, 1> (f[0], cu);
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        cu[r] = f[0][r] - cu[r];
      adj_update<R, RU, RV> (T, kHx, c, p.S, cu, nullptr, f[1], x[1], d);
      adj_far_x<R, RU, RV, 1> (f[0], cu, ERow, c.w, c.lane);
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        cu[r] = cu[r] - f[0][r];
      adj_update<R, RU, RV> (T, kHy, c, p.S, cu, nullptr, f[2], x[2], d);
    }
    if (c.source)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((c.source >> r) & 1u)
        {
          if (p.ps_on[kHx])
            f[1][r] = p.src[2 * k + 1];
          if (p.ps_on[kHy])
            f[2][r] = p.src[2 * k + 1];
        }
    }
    adj_publish<R, RU, RV, -1> (f[2], HRow, c.w, c.lane);
    __syncthreads ();
    if (probe && L.jpart && threadIdx.x == 0)
    {
      double tot = 0.0;
      for (int q = 0; q < kThreads / 32; ++q)
        tot += s_sum[q];
      adj_add (s_sum[kThreads / 32], s_sum[kThreads / 32 + 1], tot);
    }
  }
  if (probe && L.jpart && threadIdx.x == 0)
  {
    j_at ()[0] = s_sum[kThreads / 32];
    j_at ()[1] = s_sum[kThreads / 32 + 1];
  }
#pragma unroll
  for (int r = 0; r < G::C; ++r)
    if ((c.own & c.upd) >> r & 1u)
#pragma unroll
      for (int q = 0; q < 3; ++q)
      {
        out[q * N + c.id (p, r)] = f[q][r];
        if ((c.pml[q] >> r) & 1u)
          out[(3 + q) * N + c.id (p, r)] = x[q][r];
      }
}

template <typename R, int RU, int RV>
__device__ void forward_part (const Launch<R> &L, int cta, int ctas, R *S, double *s_sum)
{
  const R *in = L.load ? L.load : L.F[0];
  int to = 1;
  for (uint32_t k = L.fk0; k < L.fk1;)
  {
    // a round ends where a checkpoint is taken
    uint32_t end = min (k + (uint32_t) kRound, L.fk1);
    if (L.ck)
      end = min (end, (k / L.every + 1) * L.every);
    for (int t = cta; t < L.tiles_u * L.tiles_v; t += ctas)
    {
      __syncthreads ();   // (the shared arrays of the previous tile have been used)
      forward_tile<R, RU, RV> (L, in, L.F[to], t / L.tiles_v, t % L.tiles_v, k, (int) (end - k), S, s_sum);
    }
    if (!group_barrier (L.bar, ctas, L.err, L.limit_ns))
      return;
    in = L.F[to];
    to ^= 1;
    k = end;
  }
}

// ---- reverse group

// Transpose of component c's update on a thread's cells: a = the adjoint of F
// (in: gathered, out: of the old F), ax of X; cu gets the adjoint of the curl
// (0 on cells that are not updated).
template <typename R, int RU, int RV>
__device__ __forceinline__ void adj_transpose (const R *T, int c, const AdjCells<R, RU, RV> &cells, R S, const R *im,
                                               R a[RU * RV], R ax[RU * RV], R cu[RU * RV])
{
  using G = AdjTile<R, RU, RV>;
  if (!__any_sync (0xffffffffu, cells.pml[c]))
  {
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      cu[r] = (cells.upd >> r) & 1u ? S * (im ? im[r] : R (1)) * a[r] : R (0);
    return;
  }
  const AdjCoef<R, RU, RV> k (T, G::TM, c, RU * cells.w, RV * cells.lane);
#pragma unroll
  for (int r = 0; r < G::C; ++r)
  {
    const R m = im ? im[r] : R (1);
    const bool pm = (cells.pml[c] >> r) & 1u, up = (cells.upd >> r) & 1u;
    const R t1 = ax[r] + k.at (c, 4, r) * k.at (c, 3, r) * m * a[r];
    const R nx = k.at (c, 0, r) * t1 - k.at (c, 5, r) * k.at (c, 3, r) * m * a[r];
    cu[r] = pm ? k.at (c, 1, r) * t1 : (up ? S * m * a[r] : R (0));
    ax[r] = pm ? nx : ax[r];
    a[r] = pm ? k.at (c, 2, r) * a[r] : a[r];
  }
}

// Reverse steps k1 - 1 down to k1 - steps (all > 0) of one tile.  Ez at (x, y)
// reads Hx at y and y - 1 and Hy at x and x - 1, Hx reads Ez at y and y + 1, Hy
// at x and x + 1: the gathers below are their transposes.
template <typename R, int RU, int RV>
__device__ void reverse_tile (const Launch<R> &L, const R *in, R *out, int tu, int tv, uint32_t k1, int steps, R *S)
{
  using G = AdjTile<R, RU, RV>;
  const AdjDev<R> &p = L.p;
  const size_t N = L.N;
  const int u0 = tu * G::OU - kRound, v0 = tv * G::OV - kRound;
  R *const ZRow = S, *const YRow = S + G::A, *const T = S + 2 * G::A;
  const AdjCells<R, RU, RV> c (p, u0, v0);
  R aE[G::C], aH[2][G::C], ax[3][G::C], z[G::C], im[G::C];
  double gim[G::C];
#pragma unroll
  for (int r = 0; r < G::C; ++r)
  {
    const bool up = (c.upd >> r) & 1u;
    const int id = up ? c.id (p, r) : 0;
    aE[r] = up ? ld (in + id) : R (0);
    aH[0][r] = up ? ld (in + 2 * N + id) : R (0);
    aH[1][r] = up ? ld (in + 3 * N + id) : R (0);
    ax[kEz][r] = (c.pml[kEz] >> r) & 1u ? ld (in + N + id) : R (0);
    ax[kHx][r] = (c.pml[kHx] >> r) & 1u ? ld (in + 4 * N + id) : R (0);
    ax[kHy][r] = (c.pml[kHy] >> r) & 1u ? ld (in + 5 * N + id) : R (0);
    z[r] = up ? ld (in + 6 * N + id) : R (0);
    im[r] = up ? p.im[id] : R (0);
    gim[r] = up && ((c.own >> r) & 1u) ? L.gim[id] : 0.0;
  }
  adj_tables<R, RU, RV> (p, T, u0, v0);
  adj_publish<R, RU, RV, 1> (z, ZRow, c.w, c.lane);
  // probe cells of the thread
  unsigned probed = 0;
  const int pw = p.pr_hi[1] - p.pr_lo[1];
#pragma unroll
  for (int r = 0; r < G::C; ++r)
  {
    const int x = u0 + c.du (r), y = v0 + c.dv (r);
    probed |= ((c.upd >> r) & 1u) && x >= p.pr_lo[0] && x < p.pr_hi[0] && y >= p.pr_lo[1] && y < p.pr_hi[1] ? 1u << r : 0u;
  }
  __syncthreads ();
#pragma unroll 1
  for (int s = 0; s < steps; ++s)
  {
    const uint32_t k = k1 - 1 - s;
    const R *const dedm = L.rdedm + (size_t) (k - L.rk0) * N;
    const double *const probe = L.rprobe + (size_t) (k - L.rk0) * L.npr;
    R far[G::C], cx[G::C], cy[G::C], dm[G::C];
    // (needed after the H phase: the loads are under way meanwhile)
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      dm[r] = (c.own & c.upd) >> r & 1u ? ld (dedm + c.id (p, r)) : R (0);
    adj_far_y<R, RU, RV, 1> (z, far);
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      aH[0][r] = (c.upd >> r) & 1u ? aH[0][r] + (-z[r] + far[r]) : R (0);
    adj_far_x<R, RU, RV, 1> (z, far, ZRow, c.w, c.lane);
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      aH[1][r] = (c.upd >> r) & 1u ? aH[1][r] + (z[r] - far[r]) : R (0);
    if (c.source)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((c.source >> r) & 1u)
        {
          aH[0][r] = p.ps_on[kHx] ? R (0) : aH[0][r];
          aH[1][r] = p.ps_on[kHy] ? R (0) : aH[1][r];
        }
    }
    adj_transpose<R, RU, RV> (T, kHx, c, p.S, nullptr, aH[0], ax[kHx], cx);
    adj_transpose<R, RU, RV> (T, kHy, c, p.S, nullptr, aH[1], ax[kHy], cy);
    adj_publish<R, RU, RV, -1> (cy, YRow, c.w, c.lane);
    __syncthreads ();
    adj_far_y<R, RU, RV, -1> (cx, far);
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      cx[r] = cx[r] - far[r];
    adj_far_x<R, RU, RV, -1> (cy, far, YRow, c.w, c.lane);
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      aE[r] = (c.upd >> r) & 1u ? aE[r] + ((cx[r] + far[r]) - cy[r]) : R (0);
    if (probed)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((probed >> r) & 1u)
          aE[r] += (R) (2.0 * __ldcg (probe + (u0 + c.du (r) - p.pr_lo[0]) * pw + (v0 + c.dv (r) - p.pr_lo[1])));
    }
    if (p.ps_on[kEz] && c.source)
    {
#pragma unroll
      for (int r = 0; r < G::C; ++r)
        if ((c.source >> r) & 1u)
          aE[r] = 0;
    }
#pragma unroll
    for (int r = 0; r < G::C; ++r)
      gim[r] += (double) aE[r] * (double) dm[r];
    adj_transpose<R, RU, RV> (T, kEz, c, p.S, im, aE, ax[kEz], z);
    adj_publish<R, RU, RV, 1> (z, ZRow, c.w, c.lane);
    __syncthreads ();
  }
#pragma unroll
  for (int r = 0; r < G::C; ++r)
    if ((c.own & c.upd) >> r & 1u)
    {
      const int id = c.id (p, r);
      out[id] = aE[r];
      out[2 * N + id] = aH[0][r];
      out[3 * N + id] = aH[1][r];
      out[6 * N + id] = z[r];
      if ((c.pml[kEz] >> r) & 1u)
        out[N + id] = ax[kEz][r];
      if ((c.pml[kHx] >> r) & 1u)
        out[4 * N + id] = ax[kHx][r];
      if ((c.pml[kHy] >> r) & 1u)
        out[5 * N + id] = ax[kHy][r];
      L.gim[id] = gim[r];
    }
}

// Rounds of the reverse steps rk1 - 1 .. max (rk0, 1): the set changes with
// each.
__host__ __device__ inline int reverse_rounds (uint32_t rk0, uint32_t rk1)
{
  const uint32_t lo = rk0 > 1 ? rk0 : 1;
  return rk1 > lo ? (int) ((rk1 - lo + kRound - 1) / kRound) : 0;
}

template <typename R, int RU, int RV>
__device__ void reverse_part (const Launch<R> &L, int cta, int ctas, R *S)
{
  int cur = L.rcur;
  const uint32_t lo = L.rk0 > 1 ? L.rk0 : 1;
  for (uint32_t k = L.rk1; k > lo;)
  {
    const int steps = (int) min ((uint32_t) kRound, k - lo);
    for (int t = cta; t < L.tiles_u * L.tiles_v; t += ctas)
    {
      __syncthreads ();
      reverse_tile<R, RU, RV> (L, L.A[cur], L.A[cur ^ 1], t / L.tiles_v, t % L.tiles_v, k, steps, S);
    }
    if (!group_barrier (L.bar + kBarStride, ctas, L.err, L.limit_ns))
      return;
    cur ^= 1;
    k -= steps;
  }
}

template <typename R, int RU, int RV>
__global__ void __launch_bounds__ (kThreads, 1) adjoint_kernel (const __grid_constant__ Launch<R> L)
{
  extern __shared__ __align__ (16) unsigned char adj_smem[];
  __shared__ double s_sum[kThreads / 32 + 2];
  R *const S = reinterpret_cast<R *> (adj_smem);
  if ((int) blockIdx.x < L.fwd_ctas)
    forward_part<R, RU, RV> (L, blockIdx.x, L.fwd_ctas, S, s_sum);
  else
    reverse_part<R, RU, RV> (L, blockIdx.x - L.fwd_ctas, gridDim.x - L.fwd_ctas, S);
}

// Compensated sum of n (sum, compensation) pairs (one block of 256).
__global__ void adj_sum_kernel (const double *v, size_t n, double *acc)
{
  __shared__ double ss[256], sc[256];
  double s = 0.0, c = 0.0;
  for (size_t i = threadIdx.x; i < n; i += 256)
  {
    adj_add (s, c, v[2 * i]);
    c += v[2 * i + 1];
  }
  ss[threadIdx.x] = s;
  sc[threadIdx.x] = c;
  __syncthreads ();
  for (int o = 128; o > 0; o >>= 1)
  {
    if ((int) threadIdx.x < o)
    {
      adj_add (ss[threadIdx.x], sc[threadIdx.x], ss[threadIdx.x + o]);
      sc[threadIdx.x] += sc[threadIdx.x + o];
    }
    __syncthreads ();
  }
  if (threadIdx.x == 0)
  {
    acc[0] = ss[0];
    acc[1] = sc[0];
  }
}

// dJ/d eps from dJ/d im (gather over the Ez cells that average the cell)
template <typename R>
__global__ void grad_eps_kernel (AdjDev<R> p, const double *gim, const double *imd, int nmat, int m0x, int m0y,
                                 int m1x, int m1y, int m2x, int m2y, int m3x, int m3y, double *out)
{
  const int n = p.nx * p.ny;
  const int mx[4] = {m0x, m1x, m2x, m3x}, my[4] = {m0y, m1y, m2y, m3y};
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
  {
    const int x = t / p.ny, y = t % p.ny;
    double g = 0.0;
    for (int j = 0; j < nmat; ++j)
    {
      const int cx = x - mx[j], cy = y - my[j];
      if (cx >= 1 && cx <= p.nx - 2 && cy >= 1 && cy <= p.ny - 2)
      {
        const int c = cx * p.ny + cy;
        g -= gim[c] * imd[c] * imd[c] / (double) nmat;
      }
    }
    out[t] = g;
  }
}

// inverse averaged eps of Ez (as the per-cell kernel computes it) in R and double
template <typename R, typename E>
__global__ void invm_kernel (const E *eps, int nx, int ny, int nmat, int m1x, int m1y, int m2x, int m2y, int m3x,
                             int m3y, R *im, double *imd)
{
  const int n = nx * ny;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
  {
    const int x = t / ny, y = t % ny;
    auto at = [&] (int dx, int dy) -> E {
      const int xx = min (x + dx, nx - 1), yy = min (y + dy, ny - 1);
      return eps ? eps[xx * ny + yy] : E (1);
    };
    R m;
    double md;
    if (nmat == 2)
    {
      m = R (0.5) * ((R) at (0, 0) + (R) at (m1x, m1y));
      md = 0.5 * ((double) at (0, 0) + (double) at (m1x, m1y));
    }
    else
    {
      m = R (0.25) * ((R) at (0, 0) + (R) at (m1x, m1y) + (R) at (m2x, m2y) + (R) at (m3x, m3y));
      md = 0.25 * ((double) at (0, 0) + (double) at (m1x, m1y) + (double) at (m2x, m2y) + (double) at (m3x, m3y));
    }
    im[t] = R (1) / m;
    if (imd)
      imd[t] = 1.0 / md;
  }
}

}  // namespace

// ------------------------------------------------------------------ host side

namespace {

// One device allocation carved into 256-byte aligned pieces: reserve() every
// piece first, then allocate() once and take the pointers with at().
struct Arena
{
  std::vector<size_t> off;
  size_t total = 0;
  char *base = nullptr;
  AdjointCache *cache = nullptr;   // when set, the allocation outlives the run
  ~Arena ()
  {
    if (base && !cache)
      cudaFree (base);
  }
  template <typename Q>
  int reserve (size_t count)
  {
    off.push_back (total);
    total += (std::max<size_t> (count, 1) * sizeof (Q) + 255) & ~(size_t) 255;
    return (int) off.size () - 1;
  }
  bool allocate ()
  {
    const size_t need = std::max<size_t> (total, 256);
    if (cache && cache->base && cache->bytes >= need)
    {
      base = (char *) cache->base;
      return true;
    }
    if (cache && cache->base)
    {
      cudaFree (cache->base);
      cache->base = nullptr;
      cache->bytes = 0;
    }
    if (device_malloc ((void **) &base, need) != cudaSuccess)
      return false;
    if (cache)
    {
      cache->base = base;
      cache->bytes = need;
    }
    return true;
  }
  template <typename Q>
  Q *at (int i) const
  {
    return (Q *) (base + off[i]);
  }
};

// The kernel of a tile size (64: 64 x 64 cells in FP32, 64 x 32 in FP64; else
// 32 x 32), its own cells per tile and shared memory.
template <typename R>
const void *adjoint_pick (int tile, int &ou, int &ov, int &smem)
{
  constexpr int CV = sizeof (R) == 4 ? 2 : 1;
  if (tile == 64)
  {
    using G = AdjTile<R, 4, CV>;
    ou = G::OU;
    ov = G::OV;
    smem = G::BYTES;
    return (const void *) adjoint_kernel<R, 4, CV>;
  }
  using G = AdjTile<R, 2, 1>;
  ou = G::OU;
  ov = G::OV;
  smem = G::BYTES;
  return (const void *) adjoint_kernel<R, 2, 1>;
}

template <typename R>
cudaError_t launch (const Launch<R> &L, const void *kern, int smem, int ctas, cudaStream_t s)
{
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3 (ctas);
  lc.blockDim = dim3 (kThreads);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  lc.attrs = &attr;
  lc.numAttrs = 1;
  void *args[] = {(void *) &L};
  return cudaLaunchKernelExC (&lc, kern, args);
}

template <typename R>
std::string run_t (const Geometry &g, const void *eps_dev, bool eps_is_double, const AdjointRun &run,
                   double *objective, double *grad_host, int sm_count, cudaStream_t s)
{
  if (!g.tmz)
    return "the adjoint covers 2-D TMz grids";
  if (g.cfg.use_tfsf)
    return "the adjoint covers point-source runs (no TF/SF)";
  if (g.cfg.use_metamaterials)
    return "the adjoint does not cover metamaterials";
  const int nx = g.n[0], ny = g.n[1];
  const size_t N = (size_t) nx * ny;
  if (N > (size_t) 1 << 30)
    return "grid too large for the adjoint";
  if (run.steps < 1 || run.every < 1)
    return "steps and checkpoint interval must be positive";
  for (int a = 0; a < 2; ++a)
    if (run.probe_lo[a] < 1 || run.probe_hi[a] > g.n[a] - 1 || run.probe_lo[a] >= run.probe_hi[a])
      return "probe box outside the updated cells";
  const int npr = (run.probe_hi[0] - run.probe_lo[0]) * (run.probe_hi[1] - run.probe_lo[1]);

  // 32 x 32 tiles while half of the SMs (one group) hold them at once, else
  // the large ones, whose halo is a smaller share
  int ou = 0, ov = 0, smem = 0;
  const void *kern = adjoint_pick<R> (32, ou, ov, smem);
  if ((int64_t) ((nx + ou - 1) / ou) * ((ny + ov - 1) / ov) > sm_count / 2)
    kern = adjoint_pick<R> (64, ou, ov, smem);
  const int tiles_u = (nx + ou - 1) / ou, tiles_v = (ny + ov - 1) / ov;
  int per_sm = 0;
  if (cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor (&per_sm, kern, kThreads, smem) != cudaSuccess || per_sm < 1)
    return "the adjoint kernel does not fit on an SM";
  const int ctas = sm_count;
  const int fwd_split = std::max (1, ctas / 2);

  AdjDev<R> p{};
  p.nx = nx;
  p.ny = ny;
  const double S = 299792458.0 * g.dt / g.dx;
  p.S = (R) S;
  const int kmap[3] = {EZ, HX, HY};

  // host copies of the tables and the source values
  std::vector<std::vector<R>> tabs;
  for (int c = 0; c < 3; ++c)
  {
    const int k = kmap[c];
    const CompLayout &CL = g.comp[k];
    const int axes[3] = {CL.sig_cacb, CL.sig5, CL.sig4};
    for (int q = 0; q < 3; ++q)
      p.tax[c][q] = axes[q];
    for (int j = 0; j < 6; ++j)
    {
      std::vector<double> sg = sigma_at (g, k, axes[j / 2]);
      std::vector<R> v (sg.size ());
      for (size_t i = 0; i < sg.size (); ++i)
      {
        // the coefficient tables of the FP32 step (sigma = 0 gives 1, S, 1, 1, 1, 1)
        const double r = sg[i] * g.dt / (2 * kEps0);
        double w;
        switch (j)
        {
          case 0: w = (1 - r) / (1 + r); break;
          case 1: w = S / (1 + r); break;
          case 2: w = (1 - r) / (1 + r); break;
          case 3: w = 1 / (1 + r); break;
          case 4: w = 1 + r; break;
          default: w = 1 - r; break;
        }
        v[i] = (R) w;
      }
      tabs.push_back (std::move (v));
    }
    for (int a = 0; a < 2; ++a)
    {
      int lo = 0, hi = g.n[a];
      if (g.cfg.use_pml)
      {
        std::vector<double> sg = sigma_at (g, k, a);
        lo = 0;
        while (lo < g.n[a] && sg[lo] != 0.0)
          ++lo;
        hi = lo;
        while (hi < g.n[a] && sg[hi] == 0.0)
          ++hi;
      }
      p.ilo[c][a] = lo;
      p.ihi[c][a] = hi;
    }
  }
  // point source: E value as the E half-step writes it, H value times eta0 in
  // the stored precision
  p.ps[0] = g.cfg.point_source_mask ? g.cfg.point_source[0] : -1;
  p.ps[1] = g.cfg.point_source_mask ? g.cfg.point_source[1] : -1;
  for (int c = 0; c < 3; ++c)
    p.ps_on[c] = (g.cfg.point_source_mask >> kmap[c]) & 1;
  std::vector<R> src (2 * (size_t) run.steps);
  for (uint32_t k = 0; k < run.steps; ++k)
  {
    src[2 * k] = (R) point_source (g, k, false);
    src[2 * k + 1] = (R) point_source (g, k, true) * (R) kEta0Adj;
  }
  for (int a = 0; a < 2; ++a)
  {
    p.pr_lo[a] = run.probe_lo[a];
    p.pr_hi[a] = run.probe_hi[a];
  }

  // device memory, one allocation
  const bool grad = grad_host != nullptr;
  const uint32_t K = std::min (run.every, run.steps);
  const uint32_t nck = (run.steps + K - 1) / K;
  Arena ar;
  ar.cache = run.cache;
  std::vector<int> i_tab;
  for (const auto &v : tabs)
    i_tab.push_back (ar.reserve<R> (v.size ()));
  const int i_src = ar.reserve<R> (src.size ());
  const int i_state = ar.reserve<R> (12 * N);
  // probe tiles, and a sum per probe tile
  const int pt_u0 = run.probe_lo[0] / ou, pt_u1 = (run.probe_hi[0] - 1) / ou;
  const int pt_v0 = run.probe_lo[1] / ov, pt_v1 = (run.probe_hi[1] - 1) / ov;
  const size_t nprt = (size_t) (pt_u1 - pt_u0 + 1) * (pt_v1 - pt_v0 + 1);
  const int i_jpart = ar.reserve<double> (2 * nprt);
  const int i_im = ar.reserve<R> (N);
  const int i_imd = ar.reserve<double> (grad ? N : 0);
  const int i_acc = ar.reserve<double> (2);
  const int i_bar = ar.reserve<unsigned> (2 * kBarStride);
  const int i_err = ar.reserve<int> (1);
  int i_ck = -1, i_dedm[2] = {-1, -1}, i_probe[2] = {-1, -1}, i_adj = -1, i_gim = -1, i_gout = -1;
  if (grad)
  {
    // (the double buffers take 11 N values more than single ones would; the
    // checkpoints of the first and the last segment are not stored for that)
    i_ck = ar.reserve<R> ((size_t) (nck > 2 ? nck - 2 : 0) * 6 * N);
    for (int b = 0; b < (nck > 1 ? 2 : 1); ++b)
    {
      i_dedm[b] = ar.reserve<R> ((size_t) K * N);
      i_probe[b] = ar.reserve<double> ((size_t) K * npr);
    }
    i_adj = ar.reserve<R> (14 * N);
    i_gim = ar.reserve<double> (N);
    i_gout = ar.reserve<double> (N);
  }
  if (!ar.allocate ())
    return "device allocation failed";
  for (size_t t = 0; t < tabs.size (); ++t)
  {
    R *d = ar.at<R> (i_tab[t]);
    if (cudaMemcpyAsync (d, tabs[t].data (), tabs[t].size () * sizeof (R), cudaMemcpyHostToDevice, s) != cudaSuccess)
      return "table upload failed";
    p.tab[t / 6][t % 6] = d;
  }
  if (cudaMemcpyAsync (ar.at<R> (i_src), src.data (), src.size () * sizeof (R), cudaMemcpyHostToDevice, s) !=
      cudaSuccess)
    return "source table upload failed";
  p.src = ar.at<R> (i_src);
  R *imw = ar.at<R> (i_im);
  p.im = imw;
  R *state = ar.at<R> (i_state);
  double *acc = ar.at<double> (i_acc);
  unsigned *bar = ar.at<unsigned> (i_bar);
  int *err = ar.at<int> (i_err);
  if (cudaMemsetAsync (state, 0, 12 * N * sizeof (R), s) != cudaSuccess ||
      cudaMemsetAsync (acc, 0, 2 * sizeof (double), s) != cudaSuccess ||
      cudaMemsetAsync (ar.at<double> (i_jpart), 0, 2 * nprt * sizeof (double), s) != cudaSuccess ||
      cudaMemsetAsync (bar, 0, 2 * kBarStride * sizeof (unsigned), s) != cudaSuccess ||
      cudaMemsetAsync (err, 0, sizeof (int), s) != cudaSuccess)
    return "device initialisation failed";
  const CompLayout &LE = g.comp[EZ];
  const int blocks = (int) std::min<size_t> ((N + 255) / 256, (size_t) sm_count * 8);
  double *imd = grad ? ar.at<double> (i_imd) : nullptr;
  if (eps_is_double)
    invm_kernel<R, double><<<blocks, 256, 0, s>>> ((const double *) eps_dev, nx, ny, LE.nmat, LE.m[1][0], LE.m[1][1],
                                                   LE.m[2][0], LE.m[2][1], LE.m[3][0], LE.m[3][1], imw, imd);
  else
    invm_kernel<R, float><<<blocks, 256, 0, s>>> ((const float *) eps_dev, nx, ny, LE.nmat, LE.m[1][0], LE.m[1][1],
                                                  LE.m[2][0], LE.m[2][1], LE.m[3][0], LE.m[3][1], imw, imd);

  Launch<R> L{};
  L.p = p;
  L.N = (int) N;
  L.npr = npr;
  L.bar = bar;
  L.err = err;
  L.limit_ns = run.wait_limit_ns > 0 ? run.wait_limit_ns : kDefaultBarrierLimitNs;
  L.F[0] = state;
  L.F[1] = state + 6 * N;
  L.tiles_u = tiles_u;
  L.tiles_v = tiles_v;
  L.prt_u0 = pt_u0;
  L.prt_v0 = pt_v0;
  L.prt_nv = pt_v1 - pt_v0 + 1;

  // forward run: checkpoints, and the per-step data of the last segment
  const uint32_t last0 = (nck - 1) * K;
  L.fwd_ctas = ctas;
  L.fk0 = 0;
  L.fk1 = run.steps;
  L.jpart = ar.at<double> (i_jpart);
  L.every = K;
  if (grad)
  {
    L.ck = nck > 2 ? ar.at<R> (i_ck) : nullptr;
    L.dedm = ar.at<R> (i_dedm[0]);
    L.keep = ar.at<double> (i_probe[0]);
    L.keep0 = last0;
  }
  if (launch (L, kern, smem, ctas, s) != cudaSuccess)
    return std::string ("adjoint forward launch failed: ") + cudaGetErrorString (cudaGetLastError ());
  adj_sum_kernel<<<1, 256, 0, s>>> (L.jpart, nprt, acc);
  double hacc[2];
  int herr = 0;
  if (cudaMemcpyAsync (hacc, acc, sizeof (hacc), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync (&herr, err, sizeof (int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize (s) != cudaSuccess)
    return std::string ("forward run failed: ") + cudaGetErrorString (cudaGetLastError ());
  if (herr)
    return "a grid barrier of the adjoint forward run timed out";
  if (objective)
    *objective = hacc[0] + hacc[1];
  if (!grad)
    return "";

  // reverse sweep: launch idx reverses segment j = nck - 1 - idx from buffer
  // idx & 1 and recomputes segment j - 1 into the other buffer
  R *adj = ar.at<R> (i_adj);
  double *gim = ar.at<double> (i_gim);
  if (cudaMemsetAsync (adj, 0, 14 * N * sizeof (R), s) != cudaSuccess ||
      cudaMemsetAsync (gim, 0, N * sizeof (double), s) != cudaSuccess)
    return "device initialisation failed";
  L.A[0] = adj;
  L.A[1] = adj + 7 * N;
  L.rcur = 0;
  L.gim = gim;
  L.jpart = nullptr;
  L.ck = nullptr;
  const R *ck = ar.at<R> (i_ck);
  for (uint32_t idx = 0; idx < nck; ++idx)
  {
    const uint32_t j = nck - 1 - idx;
    const int b = (int) (idx & 1u);
    L.rk0 = j * K;
    L.rk1 = std::min (L.rk0 + K, run.steps);
    L.rdedm = ar.at<R> (i_dedm[b]);
    L.rprobe = ar.at<double> (i_probe[b]);
    if (j > 0)
    {
      L.fwd_ctas = fwd_split;
      L.fk0 = (j - 1) * K;
      L.fk1 = j * K;
      L.load = j > 1 ? ck + (size_t) (j - 2) * 6 * N : nullptr;
      // (the first segment starts from 0, in set 0)
      if (j == 1 && cudaMemsetAsync (state, 0, 6 * N * sizeof (R), s) != cudaSuccess)
        return "device initialisation failed";
      L.dedm = ar.at<R> (i_dedm[1 - b]);
      L.keep = ar.at<double> (i_probe[1 - b]);
      L.keep0 = L.fk0;
    }
    else
    {
      L.fwd_ctas = 0;
      L.load = nullptr;
      L.dedm = nullptr;
      L.keep = nullptr;
    }
    if (launch (L, kern, smem, ctas, s) != cudaSuccess)
      return std::string ("adjoint reverse launch failed: ") + cudaGetErrorString (cudaGetLastError ());
    L.rcur ^= reverse_rounds (L.rk0, L.rk1) & 1;
  }
  double *gout = ar.at<double> (i_gout);
  grad_eps_kernel<R><<<blocks, 256, 0, s>>> (p, gim, imd, LE.nmat, LE.m[0][0], LE.m[0][1], LE.m[1][0], LE.m[1][1],
                                             LE.m[2][0], LE.m[2][1], LE.m[3][0], LE.m[3][1], gout);
  if (cudaMemcpyAsync (grad_host, gout, N * sizeof (double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync (&herr, err, sizeof (int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize (s) != cudaSuccess)
    return std::string ("reverse run failed: ") + cudaGetErrorString (cudaGetLastError ());
  if (herr)
    return "a grid barrier of the adjoint reverse sweep timed out";
  return "";
}

}  // namespace

std::string adjoint_run (const Geometry &g, const void *eps_dev, bool eps_is_double, const AdjointRun &run,
                         double *objective, double *grad_host, int sm_count, cudaStream_t s)
{
  return run.fp64 ? run_t<double> (g, eps_dev, eps_is_double, run, objective, grad_host, sm_count, s)
                  : run_t<float> (g, eps_dev, eps_is_double, run, objective, grad_host, sm_count, s);
}

}  // namespace fdtdb
